"""Performance cases: the calls a user of plategpu makes, over their real range.

listed()  the named cases; draw(rng) one more case of the same ranges
prepare   the plate, its loads and the handles a program keeps (from a seed)
run       one pass through the public entry points, with its outputs
work      the bytes and operations one pass cannot do without
exact     what run returns, in 64 bits, from this file's own restatement of
          the elements and a direct solve (torch, no code of the package)

A case is a dict of plain values.  "kind" picks the call:
  solve      solveGPU on a plate whose plan is cached after its first solve
  new_mesh   solveGPU on a plate the library has not seen: partition, element
             matrices, coarse space and eigenvalue estimate included
  loads      solveGPULoadCases: several loads of one plate
  batch      Batch.solve: many uneven plates at once
  learned    Learned.solve with the committed network (144 x 144 pixels)
  train      Learned.train from given weights: forward, loss, backward, Adam
  moments    computeMoments of a displacement field
Displacements are returned as float32, as the solver interface does.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gpu-gauntlet_b200"))

import plategpu as pgp  # noqa: E402
from plategpu import _lib, learned, solver, workloads  # noqa: E402

FP64_JACOBI = {"precision": "fp64", "preconditioner": "block-jacobi", "smoother": "block-jacobi"}
FP64_TWO_LEVEL = {"precision": "fp64", "preconditioner": "two-level", "smoother": "block-jacobi"}
MIXED_CHEBYSHEV = {"precision": "mixed", "preconditioner": "two-level", "smoother": "chebyshev"}


def listed():
    return [
        # a small plate with the reference's own method: latency of the call and of one iteration
        {"name": "solve_q4_32", "kind": "solve", "mesh": "q4", "n": 32, "tol": 1e-8, **FP64_JACOBI},
        # the 60k-DOF plate with the reference's own method
        {"name": "solve_q4_141", "kind": "solve", "mesh": "q4", "n": 141, "tol": 1e-6, **FP64_JACOBI},
        # the 60k-DOF plate as the benchmark's fastest method solves it
        {"name": "solve_q4_141_mixed", "kind": "solve", "mesh": "q4", "n": 141, "tol": 3e-6, **MIXED_CHEBYSHEV},
        # a large triangle mesh of varying thickness: few iterations, much data
        {"name": "solve_dkt_200", "kind": "solve", "mesh": "dkt", "n": 200, "tol": 1e-7, **FP64_JACOBI},
        # an unstructured triangle mesh with holes and shuffled node numbers
        {"name": "solve_holes_83", "kind": "solve", "mesh": "holes", "n": 83, "tol": 2e-7, **FP64_TWO_LEVEL},
        # a plate past shared-memory capacity: the global-memory solver
        {"name": "solve_q4_400", "kind": "solve", "mesh": "q4", "n": 400, "tol": 1e-8, **FP64_TWO_LEVEL},
        # an editor's call: every solve is of a mesh not seen before
        {"name": "new_mesh_q4_141", "kind": "new_mesh", "mesh": "q4", "n": 141, "tol": 3e-6, **MIXED_CHEBYSHEV},
        # four load cases of one plate
        {"name": "loads_q4_141_x4", "kind": "loads", "mesh": "q4", "n": 141, "cases": 4, "tol": 2e-6,
         **MIXED_CHEBYSHEV},
        # many uneven plates, 70% Q4 and 30% DKT, 16 to 256 elements a side
        {"name": "batch_24", "kind": "batch", "count": 24, "low": 16, "high": 256, "mix": 5, "tol": 2e-7,
         **FP64_TWO_LEVEL},
        # the learned preconditioner inside flexible PCG
        {"name": "learned_q4_141", "kind": "learned", "mesh": "q4", "n": 141, "tol": 5e-7},
        # a few training steps of the preconditioner's network
        {"name": "train_q4_141", "kind": "train", "mesh": "q4", "n": 141, "pairs": 64, "batch": 32, "epochs": 2},
        # bending moments of a solution: the smallest call
        {"name": "moments_q4_141", "kind": "moments", "mesh": "q4", "n": 141},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "large", "new_mesh", "loads", "batch", "learned", "train", "moments"])
    if kind == "solve":
        pick = rng.choice(["jacobi", "two-level", "mixed", "dkt", "holes"])
        if pick == "mixed":  # in FP32 small plates are at the edge of stagnation: mixed is for large ones
            return {"kind": "solve", "mesh": "q4", "n": rng.randint(100, 160), "tol": 2e-6, **MIXED_CHEBYSHEV}
        if pick == "dkt":
            return {"kind": "solve", "mesh": "dkt", "n": _log_int(rng, 16, 200), "tol": 1e-7,
                    **rng.choice([FP64_JACOBI, FP64_TWO_LEVEL])}
        if pick == "holes":
            return {"kind": "solve", "mesh": "holes", "n": rng.randint(20, 90), "tol": 2e-7,
                    **rng.choice([FP64_JACOBI, FP64_TWO_LEVEL])}
        return {"kind": "solve", "mesh": "q4", "n": _log_int(rng, 8, 200), "tol": 1e-8,
                **(FP64_JACOBI if pick == "jacobi" else FP64_TWO_LEVEL)}
    if kind == "large":
        return {"kind": "solve", "mesh": "q4", "n": rng.randint(300, 400), "tol": 1e-8,
                **rng.choice([FP64_JACOBI, FP64_TWO_LEVEL, FP64_TWO_LEVEL])}
    if kind == "new_mesh":
        if rng.random() < 0.3:
            return {"kind": "new_mesh", "mesh": "dkt", "n": _log_int(rng, 16, 160), "tol": 1e-7, **FP64_JACOBI}
        return {"kind": "new_mesh", "mesh": "q4", "n": _log_int(rng, 24, 200), "tol": 1e-8, **FP64_TWO_LEVEL}
    if kind == "loads":
        return {"kind": "loads", "mesh": "q4", "n": rng.randint(100, 160), "cases": rng.randint(2, 8), "tol": 2e-6,
                **MIXED_CHEBYSHEV}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(6, 24), "low": 16, "high": rng.randint(64, 256),
                "mix": rng.randrange(1 << 20), "tol": 2e-7, **FP64_TWO_LEVEL}
    if kind == "learned":  # node grids that the committed network's 144 x 144 pixels hold
        return {"kind": "learned", "mesh": "q4", "n": rng.randint(134, 141), "tol": 5e-7 * rng.uniform(1, 2)}
    if kind == "train":
        return {"kind": "train", "mesh": "q4", "n": _log_int(rng, 40, 141), "pairs": rng.randint(32, 64),
                "batch": rng.randint(8, 32), "epochs": 2}
    return {"kind": "moments", "mesh": rng.choice(["q4", "dkt"]), "n": _log_int(rng, 16, 200)}


# --- plates -----------------------------------------------------------------

def _plate(mesh, n, seed):
    """A seeded plate of the package's own workload generators."""
    if mesh == "dkt":
        return workloads.plate_dkt_200(seed=seed, n=n)
    if mesh == "holes":
        return workloads.plate_holes_dkt(h=10.0 / n, seed=seed, q=3e3 + seed % 1000)
    if n < 64:  # all edges clamped, uniform pressure, four point loads
        return workloads.plate_q4(n, seed, edges="fixed", pressure=1e3, n_point_loads=4)
    # simply supported on the edges and on a 4 x 4 grid of columns
    return workloads.plate_q4(n, seed, edges="pinned", pressure=5e3, n_point_loads=32, column_grid=4)


def _batch_plates(case, seed):
    """Uneven plates: the sizes and element types of the case, the materials, supports and loads of the seed."""
    sizes = random.Random(case["mix"])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n = _log_int(sizes, case["low"], case["high"])
        if sizes.random() < 0.3:
            mesh = pgp.split_triangle_mesh(10.0, 10.0, n, n, jitter=0.2, seed=int(rng.integers(1 << 31)))
        else:
            mesh = pgp.mesher.rectangular_mesh_nxny(10.0, 10.0, n, n)
        material = pgp.PlateMaterial(E=float(rng.uniform(2e10, 2.1e11)), nu=float(rng.uniform(0.2, 0.3)),
                                     t=float(rng.uniform(0.05, 0.3)))
        cons = pgp.identifyConstrainedDOFs(mesh, [pgp.PlateSupport(str(rng.choice(["fixed", "pinned"])), "all_edges")])
        F = pgp.pressure_load_vector(mesh, float(rng.uniform(1e3, 1e4)))
        for node in rng.integers(0, mesh.nodeCount, size=int(rng.integers(0, 17))):
            F[3 * int(node)] += float(rng.uniform(1e3, 1e4))
        F = F.astype(np.float32)
        pgp.applyBCsToRHS(F, cons)
        out.append(workloads.Workload("plate", mesh, material, None, [], cons, F))
    return out


def _options(case):
    return pgp.GPUSolverOptions(tolerance=case["tol"], maxIterations=50000, stopRule="relative",
                                precision=case["precision"], preconditioner=case["preconditioner"],
                                smoother=case["smoother"])


def _raw_options(case):
    return solver._make_options(_options(case))


def _displacements(mesh, seed):
    """A smooth displacement field w, thx = dw/dy, thy = -dw/dx on the mesh's nodes."""
    rng = np.random.default_rng(seed)
    xy = mesh.nodes.reshape(-1, 2).astype(np.float64) * (math.pi / 10.0)
    u = np.zeros((mesh.nodeCount, 3))
    for a in range(1, 5):
        for b in range(1, 5):
            c = 1e-3 * rng.uniform(-1, 1) / (a * b)
            sx, sy, cx, cy = (f(k * xy[:, i]) for f, k, i in ((np.sin, a, 0), (np.sin, b, 1), (np.cos, a, 0),
                                                              (np.cos, b, 1)))
            u[:, 0] += c * sx * sy
            u[:, 1] += c * b * (math.pi / 10.0) * sx * cy
            u[:, 2] -= c * a * (math.pi / 10.0) * cx * sy
    return u.reshape(-1)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "batch":
        s["plates"] = _batch_plates(case, seed)
        s["loads"] = [w.F for w in s["plates"]]
        s["options"] = _raw_options(case)
        probs = [_lib.Problem(w.mesh, w.material, None, w.F, w.cons_mask) for w in s["plates"]]
        s["batch"] = solver.get_context().batch(probs, s["options"])
        return s
    w = s["plate"] = _plate(case["mesh"], case["n"], seed)
    if kind in ("solve", "new_mesh"):
        s["options"] = _options(case)
    elif kind == "loads":
        s["options"] = _options(case)
        s["loads"] = _load_cases(w, case["cases"], seed)
    elif kind == "moments":
        s["u"] = _displacements(w.mesh, seed)
    elif kind == "learned":
        s["options"] = learned.solve_options(case["tol"], 5000)
        s["solver"] = learned.LearnedSolver(solver.get_context(), w, weights=learned.DEFAULT_WEIGHTS)
    else:
        s["solver"] = ls = learned.LearnedSolver(solver.get_context(), w, seed=seed % 1000)
        s["weights"] = ls.net.get_params()
        s["pairs"] = _pairs(ls, w, case["pairs"], seed)
        s["options"] = _lib.train_options(epochs=case["epochs"], batch=case["batch"], lr=1e-3, seed=seed,
                                          loss=_lib.PG_LOSS_SCALED_L2)
    return s


def _load_cases(w, count, seed):
    """The plate's own load, then pressures with 16 point loads each."""
    rng = np.random.default_rng(seed + 1)
    loads = [w.F]
    for _ in range(count - 1):
        F = pgp.pressure_load_vector(w.mesh, float(rng.uniform(1e3, 1e4)))
        F[3 * rng.integers(0, w.mesh.nodeCount, size=16)] += rng.uniform(1e3, 1e4, size=16)
        F = F.astype(np.float32)
        pgp.applyBCsToRHS(F, w.constrainedDOFs)
        loads.append(F)
    return loads


def _pairs(ls, w, count, seed):
    """Training pairs (r, e): smooth errors e (seeded sine series, 0 on constrained DOFs) and r = K e."""
    e = torch.from_numpy(np.stack([_displacements(w.mesh, seed * 1000 + i) for i in range(count)])).cuda()
    free = torch.from_numpy(w.cons_mask == 0).cuda()
    e = (e * free).contiguous()
    zero = torch.zeros(e.shape, dtype=torch.float32, device="cuda")
    r, f = torch.empty_like(zero), torch.empty_like(zero)
    torch.cuda.synchronize()
    # make_pairs forms r = F - K x_k and e = x* - x_k; with F = 0, x* = 0 and x_k = -e: r = K e
    ls.learned.make_pairs(count, zero.data_ptr(), (e * 0).data_ptr(), (-e).contiguous().data_ptr(), r.data_ptr(),
                          f.data_ptr())
    torch.cuda.synchronize()
    return r, f


def run(s):
    kind, w = s["kind"], s.get("plate")
    if kind in ("solve", "new_mesh"):
        if kind == "new_mesh":
            pgp.clearPipelineCache()
        return pgp.solveGPU(w.mesh, w.material, w.coloring, w.F, w.constrainedDOFs, s["options"]).solution
    if kind == "loads":
        res = pgp.solveGPULoadCases(w.mesh, w.material, w.coloring, s["loads"], w.constrainedDOFs, s["options"])
        return [r.solution for r in res]
    if kind == "batch":
        xs, _, _ = s["batch"].solve(s["options"], F=s["loads"])
        return [x.astype(np.float32) for x in xs]
    if kind == "learned":
        x, _, _ = s["solver"].learned.solve(s["options"], w.F)
        return x.astype(np.float32)
    if kind == "train":
        ls, (r, e) = s["solver"], s["pairs"]
        ls.net.set_params(*s["weights"])
        ls.learned.train(r.shape[0], r.data_ptr(), e.data_ptr(), s["options"])
        p, sc = ls.net.get_params()
        return {"params": p, "scales": sc}
    return pgp.computeMoments(w.mesh, s["u"], w.material)


# --- what a pass cannot do without --------------------------------------------

def _counts(mesh, n):
    """(nodes, elements, nodes per element) of a plate."""
    if mesh == "q4":
        return (n + 1) ** 2, n * n, 4
    if mesh == "dkt":
        return (n + 1) ** 2, 2 * n * n, 3
    return int(0.97 * n * n), int(1.9 * n * n), 3


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes, tot = random.Random(case["mix"]), {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["count"]):
            n = _log_int(sizes, case["low"], case["high"])
            one = _solve_work(*_counts("dkt" if sizes.random() < 0.3 else "q4", n), 1)
            tot = {k: tot[k] + one[k] for k in tot}
        return tot
    nodes, elements, npe = _counts(case["mesh"], case["n"])
    if kind == "moments":  # mesh and displacements in, three moments out
        return {"bytes": 8 * nodes + 4 * npe * elements + 24 * nodes + 12 * nodes, "flops": 40 * elements}
    if kind == "train":  # pairs in, weights in and out; three convolution passes a training pair
        steps = case["pairs"] // min(case["batch"], case["pairs"]) * case["epochs"]
        side = (case["n"] + 1 + 2 + 7) // 8 * 8
        return {"bytes": 24 * nodes * case["pairs"] + 8 * 487008,
                "flops": 3 * learned.flops_per_image(side, side) * steps * min(case["batch"], case["pairs"])}
    return _solve_work(nodes, elements, npe, case.get("cases", 1))


def _solve_work(nodes, elements, npe, loads):
    """Mesh, supports and loads in, displacements out; the element matrices and one K x per load."""
    return {"bytes": 8 * nodes + 4 * npe * elements + 3 * nodes + loads * 24 * nodes,
            "flops": elements * (3 * npe) ** 2 * (8 + 2 * loads)}


# --- 64-bit results -------------------------------------------------------------

def _q4_matrices(c, E, nu, t):
    """Q4 Mindlin stiffness [Ne, 12, 12]: 2 x 2 Gauss bending, one-point shear (kappa = 5/6)."""
    sx, sy = c.new_tensor([-1., 1, 1, -1]), c.new_tensor([-1., -1, 1, 1])
    D = E * t ** 3 / (12 * (1 - nu ** 2))
    K = c.new_zeros(c.shape[0], 12, 12)

    def derivs(xi, eta):
        dn = torch.stack([sx * (1 + sy * eta) / 4, sy * (1 + sx * xi) / 4])  # [2, 4]
        J = torch.einsum("ak,ekb->eab", dn, c)
        return torch.linalg.solve(J, dn.expand(len(c), 2, 4)), torch.linalg.det(J).abs()

    g = 1 / math.sqrt(3.0)
    for k in range(4):
        d, det = derivs(float(sx[k]) * g, float(sy[k]) * g)
        B = c.new_zeros(c.shape[0], 3, 12)  # curvatures from thx (1::3) and thy (2::3)
        B[:, 0, 2::3], B[:, 1, 1::3] = d[:, 0], -d[:, 1]
        B[:, 2, 2::3], B[:, 2, 1::3] = d[:, 1], -d[:, 0]
        C = c.new_tensor([[1., nu, 0], [nu, 1, 0], [0, 0, (1 - nu) / 2]])
        K += torch.einsum("eia,ij,ejb,e->eab", B, C, B, det * D)
    d, det = derivs(0.0, 0.0)
    S = c.new_zeros(c.shape[0], 2, 12)
    S[:, 0, 0::3], S[:, 0, 2::3] = d[:, 0], 0.25
    S[:, 1, 0::3], S[:, 1, 1::3] = d[:, 1], -0.25
    K += torch.einsum("eia,eib,e->eab", S, S, 4 * det * (5 / 6) * E / (2 * (1 + nu)) * t)
    return K


def _dkt_matrices(c, E, nu, t):
    """DKT stiffness [Ne, 9, 9], the element as the solver defines it (three interior points)."""
    x, y = c[..., 0], c[..., 1]
    x12, x23, x31 = x[:, 0] - x[:, 1], x[:, 1] - x[:, 2], x[:, 2] - x[:, 0]
    y12, y23, y31 = y[:, 0] - y[:, 1], y[:, 1] - y[:, 2], y[:, 2] - y[:, 0]

    def side(dx, dy):  # (a, b, c, d, e) of one side
        L = dx * dx + dy * dy
        return -dx / L, 3 * dx * dy / (4 * L), (dx * dx - 2 * dy * dy) / (4 * L), -dy / L, (dy * dy - 2 * dx * dx) / (4 * L)

    (a4, b4, c4, d4, e4), (a5, b5, c5, d5, e5), (a6, b6, c6, d6, e6) = side(x23, y23), side(x31, y31), side(x12, y12)
    P4, P5, P6, t4, t5, t6 = -6 * a4, -6 * a5, -6 * a6, -6 * d4, -6 * d5, -6 * d6
    q4, q5, q6, r4, r5, r6 = 3 * a4, 3 * a5, 3 * a6, 3 * d4, 3 * d5, 3 * d6
    two_a = x12 * y31 - x31 * y12
    D = E * t ** 3 / (12 * (1 - nu ** 2))
    K = c.new_zeros(c.shape[0], 9, 9)
    for L1, L2 in ((1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3)):
        m1, m2 = 1 - 2 * L1, 1 - 2 * L2
        base = -4 + 6 * (L1 + L2)
        hx1 = [P6 * m1 + (P5 - P6) * L2, q6 * m1 - (q5 + q6) * L2, base + (c5 - c6) * L2 + c6 * m1,
               P4 * L2 + P6 * m1, q4 * L2 - q6 * m1, c4 * L2 - c6 * m1,
               -P5 * L2 - P6 * m1, q5 * L2 + q6 * m1, -c5 * L2 + c6 * m1]
        hx2 = [-P6 * m2 + (P4 - P5) * L1 - P5 * m2, q6 * m2 - (q4 + q5) * L1 + q5 * m2, base + (c4 - c5) * L1 + c5 * m2,
               P4 * m2 + P5 * L1, q4 * m2 - q5 * L1, c4 * m2 - c5 * L1,
               -P4 * L1 - P5 * m2, q4 * L1 + q5 * m2, -c4 * L1 + c5 * m2]
        hy1 = [t6 * m1 + (t5 - t6) * L2, 1 + r6 * m1 - (r5 + r6) * L2, -e6 * m1 + (b5 - b6) * L2,
               t4 * L2 + t6 * m1, -1 + r4 * L2 - r6 * m1, -e4 * L2 - b6 * m1,
               -t5 * L2 - t6 * m1, r5 * L2 + r6 * m1, e5 * L2 + b6 * m1]
        hy2 = [-t6 * m2 + (t4 - t5) * L1 - t5 * m2, 1 + r6 * m2 - (r4 + r5) * L1 + r5 * m2, e6 * m2 + (b4 - b5) * L1 - b5 * m2,
               t4 * m2 + t5 * L1, -1 + r4 * m2 - r5 * L1, -e4 * m2 + b5 * L1,
               -t4 * L1 - t5 * m2, r4 * L1 + r5 * m2, e4 * L1 - b5 * m2]
        hx1, hx2, hy1, hy2 = (torch.stack([v + 0 * x12 for v in h], 1) for h in (hx1, hx2, hy1, hy2))
        col = lambda v: v[:, None]  # noqa: E731
        B = torch.stack([-col(y23) * hx1 - col(y31) * hx2, col(x23) * hy1 + col(x31) * hy2,
                         col(x23) * hx1 + col(x31) * hx2 - col(y23) * hy1 - col(y31) * hy2], 1) / two_a[:, None, None]
        C = c.new_tensor([[1., nu, 0], [nu, 1, 0], [0, 0, (1 - nu) / 2]])
        K += torch.einsum("eia,ij,ejb,e->eab", B, C, B, two_a.abs() / 6 * D)
    return K


def _direct(w, loads):
    """[loads, 3 Nn] solutions of K u = F: block tridiagonal Cholesky over strips in y, refined twice."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m, mat = w.mesh, w.material
    xy = torch.from_numpy(m.nodes.reshape(-1, 2).astype(np.float64)).to(dev)
    el = torch.from_numpy(m.elements.reshape(-1, m.nodesPerElement).astype(np.int64)).to(dev)
    t = xy.new_full((len(el),), mat.t) if mat.elem_t is None else \
        torch.from_numpy(np.asarray(mat.elem_t, np.float64)).to(dev)
    Ke = (_q4_matrices if m.nodesPerElement == 4 else _dkt_matrices)(xy[el], mat.E, mat.nu, t)
    cons = torch.zeros(3 * m.nodeCount, dtype=torch.bool, device=dev)
    cons[torch.tensor(sorted(w.constrainedDOFs), dtype=torch.long, device=dev)] = True
    F = torch.from_numpy(np.stack(loads).astype(np.float64)).to(dev)
    F[:, cons] = 0
    # strips at least as high as any element: an element touches its strip and the next
    ye = xy[el, 1]
    height = float((ye.amax(1) - ye.amin(1)).max()) * (1 + 1e-6)
    strip = ((xy[:, 1] - xy[:, 1].min()) / height + 1e-4).floor().long()
    order = torch.argsort(strip, stable=True)
    counts = torch.bincount(strip)
    counts = [int(v) for v in counts]
    first = [0]
    for v in counts:
        first.append(first[-1] + v)
    place = torch.empty_like(order)
    place[order] = torch.arange(len(order), device=dev)
    start = torch.tensor(first, device=dev)
    dof = (3 * el[:, :, None] + torch.arange(3, device=dev)).reshape(len(el), -1)
    strip_d = strip.repeat_interleave(3)
    pos_d = (3 * (place - start[strip]))[:, None].add(torch.arange(3, device=dev)).reshape(-1)
    nd = dof.shape[1]
    r, c = dof[:, :, None].expand(-1, nd, nd).reshape(-1), dof[:, None, :].expand(-1, nd, nd).reshape(-1)
    v = Ke.reshape(-1)
    keep = ~(cons[r] | cons[c])
    r, c, v = r[keep], c[keep], v[keep]
    sr, sc = strip_d[r], strip_d[c]
    S = len(counts)
    diag, low = [], []
    by = torch.argsort(sr, stable=True)
    r, c, v, sr, sc = r[by], c[by], v[by], sr[by], sc[by]
    ends = torch.searchsorted(sr, torch.arange(S + 1, device=dev)).tolist()
    for s in range(S):
        sl = slice(ends[s], ends[s + 1])
        b = 3 * counts[s]
        A = torch.zeros(b, b, dtype=torch.float64, device=dev)
        same = sc[sl] == s
        A.index_put_((pos_d[r[sl][same]], pos_d[c[sl][same]]), v[sl][same], accumulate=True)
        nodes = order[first[s]:first[s + 1]]
        fixed = cons[(3 * nodes)[:, None].add(torch.arange(3, device=dev)).reshape(-1)]
        A += torch.diag(fixed.double())
        diag.append(A)
        if s:
            prev = sc[sl] == s - 1
            B = torch.zeros(b, 3 * counts[s - 1], dtype=torch.float64, device=dev)
            B.index_put_((pos_d[r[sl][prev]], pos_d[c[sl][prev]]), v[sl][prev], accumulate=True)
            low.append(B)
    L, G = [], []
    for s in range(S):
        A = diag[s]
        if s:
            G.append(torch.linalg.solve_triangular(L[s - 1], low[s - 1].T, upper=False).T)
            A = A - G[s - 1] @ G[s - 1].T
        L.append(torch.linalg.cholesky(A))

    def split(f):
        f = f.reshape(len(f), -1, 3)[:, order].reshape(len(f), -1)
        return [f[:, 3 * first[s]:3 * first[s + 1]].T.clone() for s in range(S)]

    def solve(b):
        for s in range(S):
            if s:
                b[s] = b[s] - G[s - 1] @ b[s - 1]
            b[s] = torch.linalg.solve_triangular(L[s], b[s], upper=False)
        for s in reversed(range(S)):
            if s + 1 < S:
                b[s] = b[s] - G[s].T @ b[s + 1]
            b[s] = torch.linalg.solve_triangular(L[s].T, b[s], upper=True)
        return b

    f = split(F)
    u = solve([a.clone() for a in f])
    for _ in range(2):
        res = []
        for s in range(S):
            a = f[s] - diag[s] @ u[s]
            if s:
                a = a - low[s - 1] @ u[s - 1]
            if s + 1 < S:
                a = a - low[s].T @ u[s + 1]
            res.append(a)
        u = [a + b for a, b in zip(u, solve(res))]
    flat = torch.cat(u).T.reshape(len(F), -1, 3)
    out = torch.empty_like(flat)
    out[:, order] = flat
    return out.reshape(len(F), -1).cpu().numpy()


def _exact_moments(w, u):
    """Nodal averages of the moments at the element centres."""
    m, mat = w.mesh, w.material
    xy, el = m.nodes.reshape(-1, 2).astype(np.float64), m.elements.reshape(-1, m.nodesPerElement).astype(np.int64)
    c = xy[el]
    if m.nodesPerElement == 4:
        dn = np.array([[-1, 1, 1, -1], [-1, -1, 1, 1]]) / 4.0
        d = np.linalg.solve(np.einsum("ak,ekb->eab", dn, c), np.broadcast_to(dn, (len(el), 2, 4)))
    else:
        two_a = (c[:, 1, 0] - c[:, 0, 0]) * (c[:, 2, 1] - c[:, 0, 1]) - (c[:, 2, 0] - c[:, 0, 0]) * (c[:, 1, 1] - c[:, 0, 1])
        nxt, prv = np.roll(c, -1, 1), np.roll(c, 1, 1)
        d = np.stack([nxt[..., 1] - prv[..., 1], prv[..., 0] - nxt[..., 0]], 1) / two_a[:, None, None]
    tx, ty = u[3 * el + 1], u[3 * el + 2]
    kx, ky = (d[:, 0] * ty).sum(1), -(d[:, 1] * tx).sum(1)
    kxy = (d[:, 1] * ty - d[:, 0] * tx).sum(1)
    D = mat.E * mat.t ** 3 / (12 * (1 - mat.nu ** 2))
    out = {}
    for name, v in (("Mx", D * (kx + mat.nu * ky)), ("My", D * (ky + mat.nu * kx)), ("Mxy", D * (1 - mat.nu) * kxy / 2)):
        s = np.bincount(el.reshape(-1), np.repeat(v, el.shape[1]), m.nodeCount)
        out[name] = s / np.maximum(1, np.bincount(el.reshape(-1), minlength=m.nodeCount))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None  # BF16 arithmetic with Adam: no 64-bit value to compare with
    if kind == "batch":
        return [_direct(w, [w.F])[0] for w in _batch_plates(case, seed)]
    w = _plate(case["mesh"], case["n"], seed)
    if kind == "moments":
        return _exact_moments(w, _displacements(w.mesh, seed))
    if kind == "loads":
        return list(_direct(w, _load_cases(w, case["cases"], seed)))
    return _direct(w, [w.F])[0]
