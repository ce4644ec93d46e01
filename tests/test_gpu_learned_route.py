"""Which way a learned solve ran, as pg_learned_stats.pdl tells it: 0 from the persistent kernel, 1 from the graph with
programmatic dependent launch (network grids past its range, and the modes without the network).  And the persistent
kernel's triangle instance against the separate kernels."""
import numpy as np
import pytest

from conftest import rel_err
from plategpu import _lib, coloring, learned, mesher, problem, workloads
from plategpu.types import PlateMaterial, PlateSupport

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, mode, pdl", [(32, _lib.LEARNED_NETWORK, 0), (230, _lib.LEARNED_NETWORK, 0),
                                          (285, _lib.LEARNED_NETWORK, 1), (32, 0, 1), (32, 2, 1)])
def test_pdl_tells_the_route(gpu_ctx, n, mode, pdl):
    wl = workloads.plate_q4(n, seed=n, edges="fixed", pressure=2e3, n_point_loads=4)
    ls = learned.LearnedSolver(gpu_ctx, wl, seed=3)
    _, _, st = ls.learned.solve(learned.solve_options(1e-8, 5), wl.F, mode)
    ls.close()
    assert st.pdl == pdl and st.mode == mode


@pytest.mark.parametrize("n", [13, 40])
def test_triangles_in_the_persistent_kernel(gpu_ctx, n):
    """Regular triangles (no jitter: their nodes are a grid).  Both solves stop at 1e-8 on the FP64 true residual."""
    m = mesher.split_triangle_mesh(10, 10, n, n, jitter=0.0, seed=1)
    sup = [PlateSupport("fixed", "all_edges")]
    cons = problem.identifyConstrainedDOFs(m, sup)
    F = problem.pressure_load_vector(m, 3e3).astype(np.float32)
    problem.applyBCsToRHS(F, cons)
    wl = workloads.Workload("dkt", m, PlateMaterial(2.1e11, 0.3, 0.1), coloring.computeElementColoringGreedy(m), sup,
                            cons, F)
    ls = learned.LearnedSolver(gpu_ctx, wl, seed=3)
    d = np.load(learned.DEFAULT_WEIGHTS)
    ls.net.set_params(d["params"], d["scales"])
    opts = learned.solve_options(1e-8, 5000)
    x, info, st = ls.learned.solve(opts, F)
    opts.phase_timing = 1
    x2, info2, st2 = ls.learned.solve(opts, F)
    ls.close()
    assert st.pdl == 0 and info.converged and info2.converged and info.true_rel_residual < 1e-8
    assert abs(info.iterations - info2.iterations) <= 1
    assert rel_err(x, x2) < 2e-6
