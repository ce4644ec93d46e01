"""Plates whose FP64 parts do not fit shared memory but whose FP32 parts do: the
method asked for runs in the persistent kernel with FP32 vectors
(pg_info.global_path 1, threads > 0), and larger ones on the global-memory
path (threads 0).  400 x 400 is the repository's configuration, 401 a ragged one,
1 x 1-block limits stay on the global-memory path."""
import numpy as np
import pytest

from conftest import rel_err
from plategpu import _lib, workloads

pytestmark = pytest.mark.gpu


def solve(ctx, wl, **kw):
    pr = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    return ctx.solve(pr, _lib.make_options(tolerance=1e-8, max_iterations=50000, stop_rule=_lib.PG_STOP_RELATIVE, **kw))


@pytest.mark.parametrize("pre", [_lib.PG_PRECOND_BLOCK_JACOBI, _lib.PG_PRECOND_TWO_LEVEL])
@pytest.mark.parametrize("n", [400, 401])
def test_fp32_layout_runs_on_the_persistent_kernel(gpu_ctx, n, pre):
    """Against an FP64-stopped solution by another route: block Jacobi over global memory (reached
    through one block fewer than the device has).  Both meet ||F - K x|| / ||F|| < 1e-8 in FP64; at that
    residual this family's solutions are within 1e-6 of the truth each, so 2e-6 of each other."""
    wl = workloads.plate_q4(n, 4, edges="pinned", pressure=5e3, n_point_loads=32, column_grid=4)
    x, info = solve(gpu_ctx, wl, preconditioner=pre)
    assert info.global_path == 1 and info.threads > 0 and info.converged and info.true_rel_residual < 1e-8
    y, ref = solve(gpu_ctx, wl, ctas=100)
    assert ref.global_path == 1 and ref.threads == 0 and ref.converged
    assert rel_err(x, y) <= 2e-6


def test_fewer_blocks_than_the_device_keep_the_global_memory_path(gpu_ctx):
    wl = workloads.plate_q4_32()
    x, info = solve(gpu_ctx, wl, ctas=1)
    assert info.global_path == 1 and info.threads == 0 and info.converged
    assert np.all(np.isfinite(x))
