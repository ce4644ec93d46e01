"""When solveGPU and its relatives read the caller's arrays in place: only while the caller is the program's one
thread.  The library runs without the interpreter lock and may wait for its context, so any other thread could write
to the arrays during the call."""
import asyncio
import threading

import numpy as np
import pytest

from plategpu import (GPUSolverOptions, _lib, computeMoments, postprocess, solveGPU, solveGPULoadCases, solver,
                      workloads)


class FakeContext:
    """Records whether the problem it was given shares the caller's arrays."""

    def __init__(self, wl):
        self.wl, self.shared = wl, []

    def _see(self, prob):
        m = self.wl.mesh
        pairs = [(prob.nodes, m.nodes), (prob.elements, m.elements), (prob.cons, self.cons)]
        if prob.F.any():
            pairs.append((prob.F, self.wl.F))
        self.shared.append([np.shares_memory(a, b) for a, b in pairs])

    def solve(self, prob, opts):
        self._see(prob)
        return np.zeros(prob.F.size), _lib.PgInfo()

    def solve_load_cases(self, prob, F, opts, width):
        self._see(prob)
        self.shared[-1].append(np.shares_memory(F, self.wl.F))
        return np.zeros(F.shape), [_lib.PgInfo() for _ in F]

    def moments(self, prob, x):
        self._see(prob)
        return tuple(np.zeros(prob.struct.node_count) for _ in range(3))


@pytest.fixture
def plate(monkeypatch):
    wl = workloads.plate_q4(6, 1)
    ctx = FakeContext(wl)
    ctx.cons = wl.cons_mask
    monkeypatch.setattr(solver, "get_context", lambda device=0: ctx)
    return wl, ctx


def calls(wl, ctx):
    solveGPU(wl.mesh, wl.material, None, wl.F, ctx.cons, GPUSolverOptions())
    solveGPULoadCases(wl.mesh, wl.material, None, [wl.F, wl.F], ctx.cons, GPUSolverOptions())
    computeMoments(wl.mesh, np.zeros(3 * wl.mesh.nodeCount), wl.material)


def test_other_threads_get_copies(plate):
    wl, ctx = plate
    stop = threading.Event()
    t = threading.Thread(target=stop.wait)
    t.start()
    try:
        calls(wl, ctx)
    finally:
        stop.set()
        t.join()
    assert ctx.shared and not any(any(s) for s in ctx.shared)


def test_async_solve_gets_copies(plate):
    wl, ctx = plate
    asyncio.run(solver.solveGPUAsync(wl.mesh, wl.material, None, wl.F, ctx.cons, GPUSolverOptions()))
    assert ctx.shared == [[False] * 4]


def test_only_thread_lends_its_arrays(plate, monkeypatch):
    wl, ctx = plate
    monkeypatch.setattr(threading, "active_count", lambda: 1)
    solveGPU(wl.mesh, wl.material, None, wl.F, ctx.cons, GPUSolverOptions())
    assert ctx.shared == [[True] * 4]
    assert postprocess.computeMoments is computeMoments
