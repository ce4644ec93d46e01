"""The row-block operator of the persistent kernel at the sizes where it can go
wrong: groups of 10 rows that are full, one row over or one short, one warp's
and several warps' groups, rows outside the registers (more than 9
neighbours; more groups than warps), parts of one node, both halo widths.

One iteration of FP64 PCG from x = 0 shows K u directly: x_1 = alpha D^-1 F with
alpha = (F, D^-1 F) / (D^-1 F, K D^-1 F).  The oracle applies K element by
element; both sum the same FP64 products in another order, at most
9 x 8 + 27 additions a row, so x_1 agrees to 1e-12 relative (about 1e4 unit
roundoffs)."""
import numpy as np
import pytest

from conftest import rel_err
from plategpu import _lib, coloring, problem, workloads
from plategpu.types import PlateMaterial, PlateMesh, PlateSupport

pytestmark = pytest.mark.gpu


def one_step(oracle, wl):
    m = wl.mesh
    ke = oracle.all_ke(m.nodes, m.elements, m.nodesPerElement, wl.material.E, wl.material.nu, wl.material.t,
                       mode=oracle.FP64, **({} if wl.material.elem_t is None else {"elem_t": wl.material.elem_t}))
    npe = m.nodesPerElement
    el = m.elements.reshape(-1, npe).astype(np.int64)
    dof = (3 * el[:, :, None] + np.arange(3)).reshape(len(el), 3 * npe)
    k = ke.reshape(len(el), 3 * npe, 3 * npe)
    free = wl.cons_mask == 0
    b = wl.F.astype(np.float64) * free
    blocks = np.zeros((m.nodeCount, 3, 3))
    for p in range(npe):
        np.add.at(blocks, el[:, p], k[:, 3 * p:3 * p + 3, 3 * p:3 * p + 3])
    f3 = free.reshape(-1, 3)
    blocks *= f3[:, :, None] & f3[:, None, :]
    blocks += np.eye(3) * ~f3[:, :, None]
    u = np.einsum("nij,nj->ni", np.linalg.inv(blocks), b.reshape(-1, 3)).reshape(-1) * free
    ku = np.zeros_like(u)
    np.add.at(ku, dof, np.einsum("eij,ej->ei", k, u[dof]))
    return u * (b @ u) / (u @ (ku * free))


def fan(spokes):
    """A hub node with `spokes` triangles around it: one row with spokes + 1 slots."""
    a = 2 * np.pi * np.arange(spokes) / spokes
    xy = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(a), np.sin(a)], 1), 2 * np.stack([np.cos(a), np.sin(a)], 1)])
    tri = []
    for i in range(spokes):
        j = (i + 1) % spokes
        tri += [(0, 1 + i, 1 + j), (1 + i, 1 + spokes + i, 1 + j), (1 + spokes + i, 1 + spokes + j, 1 + j)]
    m = PlateMesh(nodes=xy.astype(np.float32).ravel(), elements=np.asarray(tri, np.uint32).ravel(),
                  boundaryNodes=np.arange(1 + spokes, 1 + 2 * spokes, dtype=np.uint32), nodeCount=len(xy),
                  elementCount=len(tri), nodesPerElement=3)
    sup = [PlateSupport("fixed", int(k)) for k in m.boundaryNodes]
    cons = problem.identifyConstrainedDOFs(m, sup)
    F = problem.pressure_load_vector(m, 1e3).astype(np.float32)
    problem.applyBCsToRHS(F, cons)
    return workloads.Workload("fan", m, PlateMaterial(2.1e11, 0.3, 0.1), coloring.computeElementColoringGreedy(m),
                              sup, cons, F)


CASES = [(f"q4_{n}_{g}", lambda n=n: workloads.plate_q4(n, 7, pressure=1e3, n_point_loads=1), g)
         for n, g in ((2, 1), (2, 9), (3, 2), (9, 1), (9, 9), (9, 10), (9, 11), (9, 100), (12, 1), (12, 3), (25, 2),
                      (25, 4), (40, 7), (40, 148))]
CASES += [("dkt_20_3", lambda: workloads.plate_dkt_200(seed=4, n=20), 3),
          ("holes_5", lambda: workloads.plate_holes_dkt(h=0.5), 5),
          ("fan_8", lambda: fan(8), 2), ("fan_40", lambda: fan(40), 3), ("fan_200", lambda: fan(200), 4)]


@pytest.mark.parametrize("threads", [0, 32, 160, 576])
@pytest.mark.parametrize("name,make,ctas", CASES, ids=[c[0] for c in CASES])
def test_first_iterate_matches_the_oracle(gpu_ctx, oracle, name, make, ctas, threads):
    wl = make()
    pr = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    x, info = gpu_ctx.solve(pr, _lib.make_options(tolerance=1e-30, max_iterations=1, ctas=ctas, threads=threads))
    assert info.iterations == 1 and info.global_path == 0
    assert rel_err(x, one_step(oracle, wl)) < 1e-12


@pytest.mark.parametrize("threads", [0, 96, 576])
@pytest.mark.parametrize("kw", [dict(smoother=_lib.PG_SMOOTHER_CHEBYSHEV),
                                dict(preconditioner=_lib.PG_PRECOND_TWO_LEVEL),
                                dict(preconditioner=_lib.PG_PRECOND_TWO_LEVEL, smoother=_lib.PG_SMOOTHER_CHEBYSHEV)])
@pytest.mark.parametrize("precision", [_lib.PG_PREC_FP64, _lib.PG_PREC_MIXED])
@pytest.mark.parametrize("make", [lambda: fan(40), lambda: workloads.plate_q4(25, 3, n_point_loads=2)],
                         ids=["fan_40", "q4_25"])
def test_every_method_converges_to_the_truth(gpu_ctx, oracle, make, precision, kw, threads):
    """Solutions to ||r|| / ||b|| < 1e-9: 1e-6 relative error, the parity bar of the other tests."""
    wl = make()
    m = wl.mesh
    ke = oracle.all_ke(m.nodes, m.elements, m.nodesPerElement, wl.material.E, wl.material.nu, wl.material.t,
                       mode=oracle.FP64)
    xt, _ = oracle.truth_solve(m.nodeCount, m.elements, m.nodesPerElement, ke, wl.cons_mask, wl.F.astype(np.float64))
    pr = _lib.Problem(m, wl.material, wl.coloring, wl.F, wl.cons_mask)
    x, info = gpu_ctx.solve(pr, _lib.make_options(tolerance=1e-9, max_iterations=20000, ctas=5, threads=threads,
                                                  stop_rule=_lib.PG_STOP_RELATIVE, precision=precision, **kw))
    assert info.converged and rel_err(x, xt) <= 1e-6
