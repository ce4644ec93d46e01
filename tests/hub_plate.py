"""A plate one part of which touches more coarse aggregates than any regular plate's."""
import dataclasses

import numpy as np

from plategpu import _lib, mesher, problem
from plategpu.types import PlateMaterial, PlateSupport


def hub_plate(n, kites=40):
    """n x n Q4 plate (edges pinned) whose corner node also belongs to `kites` long convex quads
    that end at cells all over the plate."""
    m = mesher.rectangular_mesh_nxny(10.0, 10.0, n, n)
    rows = kites // 8
    extra = []
    for k in range(kites):
        b = (k // 8 + 1) * n // (rows + 1) * (n + 1) + (k % 8 + 1) * n // 9
        extra.append([0, b + 1, b + n + 2, b + n + 1])
    el = np.concatenate([m.elements.reshape(-1, 4), np.array(extra, np.uint32)])
    m = dataclasses.replace(m, elements=el.reshape(-1), elementCount=len(el))
    cons = problem.identifyConstrainedDOFs(m, [PlateSupport("pinned", "all_edges")])
    F = problem.pressure_load_vector(m, 5e3).astype(np.float32)
    problem.applyBCsToRHS(F, cons)
    return _lib.Problem(m, PlateMaterial(2.1e11, 0.3, 0.1), None, F, problem.constrained_mask(3 * m.nodeCount, cons))
