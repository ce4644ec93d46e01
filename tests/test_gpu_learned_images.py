"""The learned solve of plates that are small for their image: any plate's nodes may be mapped into any larger
network grid (pg_learned_create's node_pixel).  The network's work is then the image's and has to be spread as for a
plate that fills it, and the answer has to be that of the separate kernels."""
import numpy as np
import pytest

from conftest import rel_err
from plategpu import _lib, learned, workloads

pytestmark = pytest.mark.gpu


class InImage:
    """A clamped n x n plate with the committed weights in a side x side image."""

    def __init__(self, ctx, n, side):
        wl = workloads.plate_q4(n, seed=n, edges="fixed", pressure=2e3, n_point_loads=4)
        self.F = wl.F
        self.prob = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
        self.plan = ctx.plan(self.prob, _lib.make_options())
        self.net = _lib.Net(ctx, side, side, seed=3)
        d = np.load(learned.DEFAULT_WEIGHTS)
        self.net.set_params(d["params"], d["scales"])
        self.learned = _lib.Learned(self.plan, self.net, learned.grid_node_pixel(wl.mesh, side, side))

    def close(self):
        for o in (self.learned, self.net, self.plan):
            o.close()


def us_per_iteration(p):
    opts = learned.solve_options(1e-14, 40)
    infos = [p.learned.solve(opts, p.F) for _ in range(4)]
    assert all(st.network_off_at < 0 for _, _, st in infos)
    return min(1e3 * i.solve_ms / i.iterations for _, i, _ in infos)


@pytest.mark.parametrize("n, side", [(32, 144), (65, 144), (32, 272)])
def test_small_plate_costs_no_more_than_one_that_fills_the_image(gpu_ctx, n, side):
    p, full = InImage(gpu_ctx, n, side), InImage(gpu_ctx, side - 3, side)
    us, us_full = us_per_iteration(p), us_per_iteration(full)
    p.close()
    full.close()
    assert us < 1.1 * us_full, (us, us_full)


@pytest.mark.parametrize("n, side", [(7, 16), (15, 24), (15, 144), (32, 144)])
def test_small_plate_matches_separate_kernels(gpu_ctx, n, side):
    """Converged to 1e-8 on the FP64 true residual each; the bound is that of the plates that fill their image."""
    p = InImage(gpu_ctx, n, side)
    opts = learned.solve_options(1e-8, 5000)
    x, info, _ = p.learned.solve(opts, p.F)
    opts.phase_timing = 1
    x2, info2, _ = p.learned.solve(opts, p.F)
    p.close()
    assert info.converged and info2.converged and info.true_rel_residual < 1e-8
    assert rel_err(x, x2) < 2e-6
