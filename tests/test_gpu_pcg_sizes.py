"""The assembled PCG at the edges of its launch shapes: one slice, slices that are
not full, 1 to 3 (FP64) and 1 to 6 (mixed) slices an SM in shared memory and the
first size that streams, on 148 SMs; and slices of uneven width. Against the
oracle's CSR Jacobi-PCG: the FP64 loop to the same recursive tolerance (1e-10)
within one iteration; displacements of both loops within 1e-8 (max norm), the
bound of the other PCG tests. Each solve repeats its bits."""
import numpy as np
import pytest

import msolve_b200 as M
import oracle as O
from msolve_b200 import _native as N

pytestmark = pytest.mark.gpu


def check(ctx, model, E):
    mesh = M.GpuMesh(ctx, model)
    A = mesh.assemble(E, model.poisson)
    C = O.CSR(model.n_nodes, model.conn, model.dof, model.n_dofs)
    C.assemble(O.h8_stiffness_batch(model.element_xyz(), E, model.poisson)[0])
    b = model.subdomains[0].RHS
    xo, info = C.pcg_jacobi(b, tol=1e-10)
    xt, _ = C.pcg_jacobi(b, tol=1e-13)
    # (one element under a uniform load is solved exactly in one iteration, after
    # which the mixed loop's FP32 recursion has nothing left to reduce and breaks down)
    for precision in ("fp64", "mixed") if model.n_elems > 1 else ("fp64",):
        s = M.SolverPCG(ctx, model, 20000, 1e-10, precision)
        s.matrix = A
        x = s.Solve().copy()
        assert np.abs(x - xt).max() <= 1e-8 * np.abs(xt).max(), precision
        if precision == "fp64":
            assert abs(s.iterations - info["iterations"]) <= 1
            assert np.abs(x - xo).max() <= 1e-9 * np.abs(xo).max()
        assert np.array_equal(x, s.Solve()), precision


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (3, 3, 1), (10, 4, 4), (15, 16, 16), (16, 16, 17), (21, 20, 21),
                                      (24, 24, 24), (27, 27, 26), (29, 29, 28), (31, 31, 30)])
def test_pcg_launch_shapes(ctx, nx, ny, nz):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    check(ctx, model, np.exp(0.3 * np.random.default_rng(nx).standard_normal(model.n_elems)))


def test_pcg_uneven_slices(ctx):
    """Nodes numbered at random: the rows of a slice have 8 to 27 blocks."""
    m0 = M.clamped_block_model(9, ny=8, nz=7)
    p = np.random.default_rng(2).permutation(m0.n_nodes)
    model = M.Model(m0.xyz[np.argsort(p)], p[m0.conn], 1.0, 0.3)
    model.constrain(np.nonzero(model.xyz[:, 2] == 0.0)[0])
    for n in np.nonzero(model.xyz[:, 2] == 7.0)[0]:
        model.add_load(n, 2, -1.0)
    model.ConnectDataStructures()
    check(ctx, model, np.exp(0.3 * np.random.default_rng(3).standard_normal(model.n_elems)))


def test_pcg_streams_at_full_size(ctx):
    """A matrix past L2 (evict-first loads): mixed and FP64 agree to 1e-8."""
    model = M.clamped_block_model(44, ny=44, nz=40)
    A = M.GpuMesh(ctx, model).assemble(np.exp(0.3 * np.random.default_rng(4).standard_normal(model.n_elems)), 0.3)
    x = []
    for precision in ("fp64", "mixed"):
        s = M.SolverPCG(ctx, model, 20000, 1e-11, precision)
        s.matrix = A
        x.append(s.Solve().copy())
    b = model.subdomains[0].RHS
    assert np.linalg.norm(b - A.Multiply(x[0])) <= 1e-9 * np.linalg.norm(b)
    assert np.abs(x[0] - x[1]).max() <= 1e-8 * np.abs(x[0]).max()


# the largest matrices of one and two slices an SM on a third of 148 SMs and the next
# ones (FP64), of six (mixed), and the first sizes of 4, 2 and 1 warps a slice
@pytest.mark.parametrize("nx,ny,nz", [(11, 11, 10), (13, 13, 15), (14, 13, 14), (16, 15, 16), (20, 20, 20), (20, 21, 20),
                                      (25, 24, 24), (37, 22, 29), (40, 40, 37)])
def test_pcg_rule_edges(ctx, nx, ny, nz):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    check(ctx, model, np.exp(0.3 * np.random.default_rng(nx).standard_normal(model.n_elems)))


def test_pcg_several_rounds_of_slices(ctx):
    """More slices than a launch's CTAs take at a time: mixed and FP64 agree to 1e-8."""
    model = M.clamped_block_model(53, ny=53, nz=52)
    A = M.GpuMesh(ctx, model).assemble(np.exp(0.3 * np.random.default_rng(5).standard_normal(model.n_elems)), 0.3)
    x = []
    for precision in ("fp64", "mixed"):
        s = M.SolverPCG(ctx, model, 20000, 1e-11, precision)
        s.matrix = A
        x.append(s.Solve().copy())
        assert np.array_equal(x[-1], s.Solve()), precision
    b = model.subdomains[0].RHS
    assert np.linalg.norm(b - A.Multiply(x[0])) <= 1e-9 * np.linalg.norm(b)
    assert np.abs(x[0] - x[1]).max() <= 1e-8 * np.abs(x[0]).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [6, 18, 26])
def test_pcg_limits(ctx, n, precision):
    """A limit below, at and above a round of launches: the count is the limit."""
    model = M.clamped_block_model(n)
    A = M.GpuMesh(ctx, model).assemble(np.exp(0.3 * np.random.default_rng(1).standard_normal(model.n_elems)), 0.3)
    for limit in (1, 2, 5, 70):
        s = M.SolverPCG(ctx, model, limit, 1e-12, precision)
        s.matrix = A
        with pytest.raises(M.InvalidOperationError) as e:
            s.Solve()
        assert e.value.code == N.MSG_ERR_NOT_CONVERGED and s.iterations == limit
