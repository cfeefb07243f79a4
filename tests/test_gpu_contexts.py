"""Contexts on host threads of their own, solving at the same time: every call
gives the status and the bits of the same call alone."""
import ctypes as C
import threading

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
