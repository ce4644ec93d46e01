"""How long a mixed two-level solve keeps going while its FP64 residual is flat: with the automatic interval of 50
updates, for 300.  These thin plates' residuals stay flat for more than 150 updates and then fall below the tolerance;
each must converge without the FP64 correction, by one load and by load cases in lockstep.  Three replacements at a
caller's own interval of 50 still end the solve."""
import numpy as np
import pytest

from plategpu import _lib, mesher, problem
from plategpu.types import PlateMaterial, PlateSupport

pytestmark = pytest.mark.gpu


def thin_plate(nx, ny, t, edges, cols):
    m = mesher.rectangular_mesh_nxny(10.0, 10.0 * ny / nx, nx, ny)
    sup = [PlateSupport(edges, "all_edges")]
    for a in range(cols):
        for b in range(cols):
            i, j = round((a + 1) * nx / (cols + 1)), max(1, round((b + 1) * ny / (cols + 1)))
            sup.append(PlateSupport("pinned", j * (nx + 1) + i))
    cons = problem.identifyConstrainedDOFs(m, sup)
    F = problem.pressure_load_vector(m, 5e3).astype(np.float32)
    problem.applyBCsToRHS(F, cons)
    return _lib.Problem(m, PlateMaterial(2.1e11, 0.3, t), None, F, problem.constrained_mask(3 * m.nodeCount, cons))


def options(**kw):
    return _lib.make_options(tolerance=2e-6, max_iterations=8000, stop_rule=_lib.PG_STOP_RELATIVE, fallback=0,
                             precision=_lib.PG_PREC_MIXED, preconditioner=_lib.PG_PRECOND_TWO_LEVEL, **kw)


@pytest.mark.parametrize("nx, ny, t, edges, cols", [(32, 32, 0.02, "pinned", 3), (32, 32, 0.02, "pinned", 4),
                                                    (48, 12, 0.01, "fixed", 4)])
def test_flat_residual_is_waited_for(gpu_ctx, nx, ny, t, edges, cols):
    prob = thin_plate(nx, ny, t, edges, cols)
    _, info = gpu_ctx.solve(prob, options())
    _, infos = gpu_ctx.solve_load_cases(prob, np.stack([prob.F, 0.5 * prob.F]), options())
    for i in (info, *infos):
        assert i.converged and i.fallback == 0 and i.true_rel_residual < 2e-6
    _, own = gpu_ctx.solve(prob, options(reliable_interval=50))
    assert own.stop_reason == _lib.PG_STOP_STAGNATED
