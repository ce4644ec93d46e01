"""Which kernel a plate near shared-memory capacity gets: the same at the first call, which builds the coarse space,
and at every later one, and never a refusal where another path is left.

About 325 elements a side is where FP64 two-level parts stop fitting (the row blocks then run with FP32 vectors), 359
where block-Jacobi ones do.  In the hub plate one part touches more than 25 aggregates."""
import numpy as np
import pytest

from conftest import rel_err
from hub_plate import hub_plate
from plategpu import _lib, workloads

pytestmark = pytest.mark.gpu

TL = _lib.PG_PRECOND_TWO_LEVEL


def options(**kw):
    return _lib.make_options(stop_rule=_lib.PG_STOP_RELATIVE, **kw)


@pytest.mark.parametrize("n, pre", [(323, TL), (324, TL), (325, TL), (326, TL), (358, 0), (359, 0), (360, 0)])
def test_first_and_later_calls_take_one_path(gpu_ctx, n, pre):
    wl = workloads.plate_q4(n, 4, edges="pinned", pressure=5e3, n_point_loads=32, column_grid=4)
    prob = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    gpu_ctx.clear_cache()
    calls = [gpu_ctx.solve(prob, options(tolerance=1e-6, max_iterations=30, preconditioner=pre))[1] for _ in range(3)]
    assert calls[0].plan_cached == 0 and calls[1].plan_cached == 1
    keys = [(i.global_path, i.threads, i.shared_bytes, i.iterations) for i in calls]
    assert keys[0] == keys[1] == keys[2]
    assert keys[0][1] > 0


@pytest.mark.parametrize("n", [306, 308, 310, 312])
def test_part_that_touches_many_aggregates(gpu_ctx, n):
    prob = hub_plate(n)
    gpu_ctx.clear_cache()
    calls = [gpu_ctx.solve(prob, options(tolerance=1e-6, max_iterations=30, preconditioner=TL))[1] for _ in range(2)]
    assert [(i.global_path, i.threads) for i in calls[:1]] == [(i.global_path, i.threads) for i in calls[1:]]
    assert calls[0].iterations == 30


@pytest.mark.parametrize("n", [326, 360])
def test_fp32_vectors_just_past_fp64_capacity(gpu_ctx, n):
    """Against block Jacobi over global memory (one block fewer than the device has); both stop at 1e-8 on the
    FP64 true residual, where this family's solutions are within 1e-6 of the truth each."""
    wl = workloads.plate_q4(n, 4, edges="pinned", pressure=5e3, n_point_loads=32, column_grid=4)
    prob = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    x, info = gpu_ctx.solve(prob, options(tolerance=1e-8, max_iterations=50000, preconditioner=TL))
    assert info.global_path == 1 and info.threads > 0 and info.converged and info.true_rel_residual < 1e-8
    y, ref = gpu_ctx.solve(prob, options(tolerance=1e-8, max_iterations=50000, ctas=100))
    assert ref.global_path == 1 and ref.threads == 0 and ref.converged
    assert rel_err(x, y) <= 2e-6
