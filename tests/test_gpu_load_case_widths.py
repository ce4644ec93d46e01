"""Load-case launches of different widths on one plan: their buffers serve every width, so a call of 4 + 2 cases
costs less than one of 4 + 4, and neither changes what the other returns."""
import time

import numpy as np
import pytest

from plategpu import _lib, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plate():
    wl = workloads.plate_q4_141()
    F = np.stack([wl.F * np.float32(1 + 0.1 * k) for k in range(8)])
    return _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask), F


@pytest.mark.parametrize("precision", [_lib.PG_PREC_FP64, _lib.PG_PREC_MIXED])
def test_widths_share_their_buffers(gpu_ctx, plate, precision):
    prob, F = plate
    opts = _lib.make_options(tolerance=2e-6, max_iterations=20000, stop_rule=_lib.PG_STOP_RELATIVE,
                             precision=precision, preconditioner=_lib.PG_PRECOND_TWO_LEVEL)

    def call(count, width=0):
        t = time.perf_counter()
        X, _ = gpu_ctx.solve_load_cases(prob, F[:count], opts, width)
        return time.perf_counter() - t, X

    first = {c: call(c)[1] for c in (8, 6, 2)}
    pair = call(2, 2)[1]
    ms = {c: min(call(c)[0] for _ in range(5)) for c in (6, 8)}
    for c in (2, 8, 6):
        np.testing.assert_array_equal(call(c)[1], first[c])
    np.testing.assert_array_equal(call(2, 2)[1], pair)
    np.testing.assert_array_equal(first[6][:4], first[8][:4])
    assert ms[6] < ms[8], ms  # two cases less
