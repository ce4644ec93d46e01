"""FP64 requests past FP64 shared-memory capacity: what is left of the FP32 attempt when it gives up and the
global-memory path runs, and that the options of mixed solves have no say in it."""
import numpy as np
import pytest

from plategpu import _lib, workloads

pytestmark = pytest.mark.gpu

N = 400
TWO_LEVEL = dict(preconditioner=_lib.PG_PRECOND_TWO_LEVEL)


def solve(ctx, wl, **kw):
    pr = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    return ctx.solve(pr, _lib.make_options(tolerance=1e-8, stop_rule=_lib.PG_STOP_RELATIVE, **kw))


@pytest.mark.parametrize("method", [TWO_LEVEL, {}], ids=["two-level", "block-jacobi"])
def test_record_after_a_stalled_attempt(gpu_ctx, method):
    """A plate too thin for FP32 (condition number times its epsilon far above 1): the attempt stalls, the
    global-memory path ends at the iteration limit.  Its record is that path's, the time that of both: what the
    call took beyond solve_ms (staging, launches) is far below the attempt's 800 updates of about 20 us."""
    wl = workloads.plate_q4(N, 4, edges="fixed", pressure=5e3, n_point_loads=4, t=0.001)
    for call in range(2):  # the second one without set-up
        _, info = solve(gpu_ctx, wl, max_iterations=1500, **method)
    assert info.global_path == 1 and info.stop_reason == _lib.PG_STOP_MAX_ITER and info.iterations == 1500
    assert (info.threads, info.shared_bytes, info.coarse_dim, info.fallback) == (0, 0, 0, 0)
    assert info.setup_ms == 0.0 and info.coarse_ms == 0.0 and info.plan_ms == 0.0
    assert info.total_ms - info.solve_ms < 8.0


def test_mixed_options_have_no_say(gpu_ctx):
    wl = workloads.plate_q4(N, 4, edges="pinned", pressure=5e3, n_point_loads=32, column_grid=4)
    plain = solve(gpu_ctx, wl, max_iterations=50000, **TWO_LEVEL)
    for kw in (dict(reliable_interval=10), dict(reliable_interval=1000), dict(reliable_delta=0.5)):
        x, info = solve(gpu_ctx, wl, max_iterations=50000, **TWO_LEVEL, **kw)
        assert info.converged and info.global_path == 1 and info.threads > 0
        assert info.reliable_updates == plain[1].reliable_updates
        np.testing.assert_array_equal(x, plain[0])
