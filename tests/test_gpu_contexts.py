"""Contexts on host threads of their own, solving at the same time: every call
gives the status and the bits of the same call alone."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

import msolve_b200 as M
from msolve_b200 import _native as N

pytestmark = pytest.mark.gpu
CALLS = 4000
ITERATIONS = 2  # a call is short, so that the threads' launches meet often


class Assembled:
    """A matrix on a context of its own, at most one slice of 32 rows an SM: a layer
    one element thick has 18 blocks a row, a block 27."""

    def __init__(self, nx, ny, nz, precision):
        self.ctx = M.Context(0)
        model = M.clamped_block_model(nx, ny=ny, nz=nz)
        self.matrix = M.GpuMesh(self.ctx, model).assemble(np.linspace(0.5, 2.0, model.n_elems), 0.3)
        self.b = N.f64(model.subdomains[0].RHS)
        self.fn = N.lib().MSG_PCG_SOLVE_MIXED if precision == "mixed" else N.lib().MSG_PCG_SOLVE

    def solve(self):
        x, it, rr = np.zeros(self.b.size), C.c_int(0), C.c_double(0)
        st = self.fn(self.matrix.handle, N.ptr(self.b), N.ptr(x), ITERATIONS, 1e-10, C.byref(it), C.byref(rr))
        return st, x


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_matrices_of_other_widths_side_by_side(precision):
    systems = [Assembled(*sides, precision) for sides in ((15, 15, 1), (7, 7, 7)) * 2]
    alone = [s.solve() for s in systems]
    assert all(st == N.MSG_ERR_NOT_CONVERGED for st, _ in alone)
    failed = []
    start = threading.Barrier(len(systems))

    def work(s, x0):
        start.wait()
        for _ in range(CALLS):
            st, x = s.solve()
            if st != N.MSG_ERR_NOT_CONVERGED or not np.array_equal(x, x0):
                failed.append((st, N.lib().MSG_LAST_ERROR(s.ctx.handle)))
                return

    threads = [threading.Thread(target=work, args=(s, x)) for s, (_, x) in zip(systems, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("n,precision", [(44, "fp64"), (44, "mixed"), (20, "fp64")])
def test_a_solve_leaves_room_for_other_contexts(n, precision):
    """Small solves and a batch beside solves that could fill the device take a fraction
    of one of those, not its whole time for each launch that has to wait for its end.
    (A 24^3 x 64 batch is some hundred launches of the whole device.)"""
    ctx = M.Context(0)
    model = M.clamped_block_model(n)
    big = M.SolverPCG(ctx, model, 20000, 1e-10, precision)
    big.matrix = M.GpuMesh(ctx, model).assemble(np.linspace(0.5, 2.0, model.n_elems), 0.3)

    small_ctx = M.Context(0)
    cantilever = M.cantilever_model()
    small = M.SolverPCG(small_ctx, cantilever, 20000, 1e-7)
    small.matrix = M.GpuMesh(small_ctx, cantilever).assemble(np.ones(cantilever.n_elems), 0.3)
    block = M.clamped_block_model(24)
    kl = M.LognormalStochasticCoefficientsProvider([24] * 3, 6.0, 10, 6)
    batch = M.MonteCarloAnalyzerWithStochasticMaterial(small_ctx, block, kl, expansion_order=10, simulations=64, seed=1,
                                                       mode="mixed", tolerance=1e-10, keep_solutions=False)
    batch.Initialize()

    def median(f, calls):
        f()
        t = []
        for _ in range(calls):
            t0 = time.perf_counter()
            f()
            t.append(time.perf_counter() - t0)
        return sorted(t)[calls // 2]

    alone = median(big.Solve, 5), median(small.Solve, 9), median(batch.Solve, 5)
    stop = threading.Event()

    def loop():
        while not stop.is_set():
            big.Solve()

    t = threading.Thread(target=loop)
    t.start()
    try:
        beside = median(small.Solve, 9), median(batch.Solve, 5)
    finally:
        stop.set()
        t.join()
    # a small solve's one launch never waits for the end of a big solve; the batch gets
    # at least a quarter of the device
    assert beside[0] <= alone[1] + 0.4 * alone[0], (alone, beside)
    assert beside[1] <= 4.0 * alone[2], (alone, beside)
