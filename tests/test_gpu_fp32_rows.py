"""FP32 rows of K: mixed solves of clamped plates, whose lowest modes an FP32 product resolves only when
a translation in w leaves no rounding behind.

A replacement interval of 200 updates leaves the FP32 product alone for most of a solve.  Each solve must meet
its tolerance on the FP64 true residual, without the FP64 correction, by one load, by load cases in lockstep and in a
batch; the solution's bound is the repository's for this stop, 1e-6 relative at tolerance 1e-6 on these plates (their
condition number times the residual, over the smooth part that the load excites), against an FP64 solve."""
import numpy as np
import pytest

from conftest import rel_err
from plategpu import _lib, workloads

pytestmark = pytest.mark.gpu

MIXED = dict(precision=_lib.PG_PREC_MIXED, preconditioner=_lib.PG_PRECOND_TWO_LEVEL,
             smoother=_lib.PG_SMOOTHER_CHEBYSHEV, reliable_interval=200, fallback=0)


def options(**kw):
    return _lib.make_options(tolerance=1e-6, max_iterations=20000, stop_rule=_lib.PG_STOP_RELATIVE, **kw)


@pytest.mark.parametrize("n", [48, 100, 141])
def test_clamped_plate_converges_in_mixed_precision(gpu_ctx, n):
    wl = workloads.plate_q4(n, 3, edges="fixed", pressure=5e3, n_point_loads=32)
    prob = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    truth, _ = gpu_ctx.solve(prob, _lib.make_options(tolerance=1e-11, max_iterations=20000,
                                                     stop_rule=_lib.PG_STOP_RELATIVE,
                                                     preconditioner=_lib.PG_PRECOND_TWO_LEVEL))
    opts = options(**MIXED)
    x, info = gpu_ctx.solve(prob, opts)
    X, infos = gpu_ctx.solve_load_cases(prob, np.stack([wl.F, 0.5 * wl.F]), opts)
    b = gpu_ctx.batch([prob], opts)
    xb, infob, _ = b.solve(opts)
    b.close()
    for got, i in ((x, info), (X[0], infos[0]), (2.0 * X[1], infos[1]), (xb[0], infob[0])):
        assert i.converged and i.fallback == 0 and i.true_rel_residual < 1e-6
        assert rel_err(got, truth) < 1e-6
