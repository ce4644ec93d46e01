"""The batch schedule that pg_batch_schedule tells (batch_part_nodes = 400) is the one a batch with that option runs."""
import numpy as np
import pytest

from plategpu import _lib, workloads

pytestmark = pytest.mark.gpu


def test_schedule_is_the_batch_s(gpu_ctx):
    sides = [16, 31, 48, 64, 100, 127, 150, 31]
    probs = []
    for n in sides:
        wl = workloads.plate_q4(n, n)
        probs.append(_lib.Problem(wl.mesh, wl.material, None, wl.F, wl.cons_mask))
    opts = _lib.make_options(tolerance=1e-2, max_iterations=3, preconditioner=_lib.PG_PRECOND_TWO_LEVEL,
                             batch_part_nodes=400)
    b = gpu_ctx.batch(probs, opts)
    _, infos, bi = b.solve(opts)
    b.close()
    told = _lib.batch_schedule([(n + 1) ** 2 for n in sides], 148, 450)
    np.testing.assert_array_equal([i.ctas for i in infos], told["plate_size"])
    assert (bi.phases, bi.grid) == (told["phases"], max(told["phase_grid"]))
