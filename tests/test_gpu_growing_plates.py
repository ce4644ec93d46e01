"""Plans of ever larger plates cost what plans of plates already seen do: no host buffer is made anew for each."""
import statistics

import pytest

from plategpu import _lib, workloads

pytestmark = pytest.mark.gpu


def test_growing_plates_reuse_the_staging():
    probs = []
    for n in range(122, 162, 2):
        wl = workloads.plate_q4(n, n, edges="pinned", pressure=5e3)
        probs.append(_lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask))
    opts = _lib.make_options(tolerance=1e-3, max_iterations=1)
    ctx = _lib.Context(0)

    def plans():
        out = []
        for p in probs:
            _, info = ctx.solve(p, opts)
            assert info.plan_cached == 0
            out.append(info.plan_ms)
        ctx.clear_cache()
        return statistics.median(out)

    growing, known = plans(), plans()
    ctx.close()
    assert growing < 1.4 * known, (growing, known)
