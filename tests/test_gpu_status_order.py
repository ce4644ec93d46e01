"""Status of a call with two faults: the problem's own (PG_EINVAL) comes before its load's (PG_ENONFINITE), on a mesh
the library has not seen and on one whose valid twin is cached."""
import numpy as np
import pytest

from plategpu import PlateGPUError, _lib, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", ["element", "node", "thickness"])
@pytest.mark.parametrize("cached", [False, True])
def test_invalid_problem_with_nonfinite_load(gpu_ctx, bad, cached):
    wl = workloads.plate_q4(8, 1)
    prob = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    prob.elem_t = np.full(wl.mesh.elementCount, 0.1, np.float32)
    prob.struct.elem_t = prob.elem_t.ctypes.data
    opts = _lib.make_options()
    gpu_ctx.clear_cache()
    if cached:
        gpu_ctx.solve(prob, opts)
    prob.F[5] = np.nan
    with pytest.raises(PlateGPUError) as e:  # the load alone
        gpu_ctx.solve(prob, opts)
    assert e.value.status == "PG_ENONFINITE"
    if bad == "element":
        prob.elements[3] = wl.mesh.nodeCount
    elif bad == "node":
        prob.nodes[7] = np.inf
    else:
        prob.elem_t[2] = np.nan
    for call in (lambda: gpu_ctx.solve(prob, opts), lambda: gpu_ctx.solve_load_cases(prob, np.stack([prob.F] * 2), opts)):
        with pytest.raises(PlateGPUError) as e:
            call()
        assert e.value.status == "PG_EINVAL"
