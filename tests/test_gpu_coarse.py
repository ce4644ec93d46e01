"""The coarse inverse by 32-mode elimination steps at the edges of its tiles, and
the eigenvalue estimate from the row blocks, against the numpy model of both
(two_level_ref).  C = 3 ctas: 3, 30, 33, 63, 66, 96, 99, 129, 300 modes fill one
tile in part, one row over a tile, one short of two, and so on."""
import numpy as np
import pytest

from plategpu import _lib, workloads
from test_gpu_two_level import fp64_operator
from two_level_ref import coarse_basis, lambda_max_power, strip_partition, two_level_pcg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 10, 11, 21, 22, 32, 33, 43, 100])
def test_iterations_match_the_model_at_tile_edges(gpu_ctx, oracle, ctas):
    """The count of iterations to 1e-8 within 3% + 2 of the model's (the bar of the other two-level
    tests): a wrong or dropped entry of A_c^-1 changes it by far more, or breaks convergence."""
    wl = workloads.plate_q4(25, 3, edges="pinned", n_point_loads=3, column_grid=2)
    _ke, A, bd, b = fp64_operator(oracle, wl)
    xy = wl.mesh.nodes.reshape(-1, 2).astype(np.float64)
    P = coarse_basis(xy, wl.cons_mask, strip_partition(xy, ctas), ctas)
    _x, model = two_level_pcg(A, b, bd, P, 1e-8)
    pr = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    x, info = gpu_ctx.solve(pr, _lib.make_options(tolerance=1e-8, max_iterations=20000, ctas=ctas,
                                                  stop_rule=_lib.PG_STOP_RELATIVE,
                                                  preconditioner=_lib.PG_PRECOND_TWO_LEVEL))
    assert info.converged and info.coarse_dim == 3 * ctas
    assert abs(info.iterations - model) <= 0.03 * model + 2


@pytest.mark.parametrize("make", [lambda: workloads.plate_q4(9, 3), lambda: workloads.plate_dkt_200(seed=2, n=17),
                                  lambda: workloads.plate_holes_dkt(h=0.6)], ids=["q4_9", "dkt_17", "holes"])
def test_lambda_max_matches_the_model(gpu_ctx, oracle, make):
    """30 power steps in FP64 in another order of additions: 1e-10 relative (rounding of 30 steps of
    about 100 terms, 30 x 100 x 1.1e-16 = 3e-13, grows at most a hundredfold here)."""
    wl = make()
    _ke, A, bd, _b = fp64_operator(oracle, wl)
    pr = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    _x, info = gpu_ctx.solve(pr, _lib.make_options(tolerance=1e-6, max_iterations=20000, ctas=3,
                                                   stop_rule=_lib.PG_STOP_RELATIVE,
                                                   smoother=_lib.PG_SMOOTHER_CHEBYSHEV))
    lam = lambda_max_power(A, bd, wl.cons_mask)
    assert abs(info.smoother_lambda_max - lam) <= 1e-10 * lam
