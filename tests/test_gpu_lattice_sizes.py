"""Batched mixed solves on lattices whose sides are not multiples of the
operators' tiles: displacements against FP64 oracle solves (1e-13 recursive
residual). The mixed solve stops at a true residual of 1e-10; its displacement
error on these blocks stays below 1e-10 times the condition number's square
root (under 100), so 1e-8 (max norm) is the bound, as in the other parity
tests."""
import numpy as np
import pytest

import msolve_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


def solve_and_compare(ctx, nx, ny, nz, R, K=12, sigma=0.3, tol=1e-10):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    L = [nx, ny, nz]
    kl = M.LognormalStochasticCoefficientsProvider(L, 0.3 * nx, K, 8, sigma=sigma)
    mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=K, simulations=R, seed=nx + ny + nz,
                                                    mode="mixed", tolerance=tol)
    mc.Initialize()
    mc.Solve()
    rows = sorted({0, R // 2, R - 1})
    E = O.kl_field(O.centroids(model.xyz, model.conn), L, kl.table(), mc.RandomNumbers[rows], sigma=sigma)
    cons = (model.dof < 0).astype(np.uint8)
    for i, r in enumerate(rows):
        xo, _ = O.block_solve_pcg(nx, ny, nz, cons, E[i], model.poisson, model.subdomains[0].RHS, tol=1e-13)
        assert np.abs(mc.Solutions[r] - xo).max() <= 1e-8 * np.abs(xo).max(), (r, nx, ny, nz)
    return mc


# nodes across a tile of 7 x 3 node pencils: one short, exact, one more, in y and z
@pytest.mark.parametrize("nx,ny,nz,R", [(4, 4, 4, 3), (6, 6, 4, 17), (4, 8, 8, 64), (8, 12, 6, 65), (10, 14, 10, 16)])
def test_tile_edges(ctx, nx, ny, nz, R):
    solve_and_compare(ctx, nx, ny, nz, R)


# odd axes: levels whose last element is half empty, alone and after even ones;
# the smallest lattices of the rule and the largest of the Jacobi loop; thin and tall
@pytest.mark.parametrize("nx,ny,nz,R", [(5, 5, 5, 7), (3, 9, 8, 33), (7, 7, 7, 64), (9, 15, 6, 20), (10, 12, 11, 65),
                                        (21, 13, 9, 3), (5, 5, 20, 8), (12, 12, 5, 17)])
def test_odd_axes(ctx, nx, ny, nz, R):
    solve_and_compare(ctx, nx, ny, nz, R)


@pytest.mark.parametrize("sigma", [0.8, 1.2])
def test_odd_axes_strong_contrast(ctx, sigma):
    """The odd lattices' damping holds for any positive field (they ran by Jacobi
    before they coarsened): moduli over three decades. Residual 1e-12, since the
    condition number grows with the contrast."""
    solve_and_compare(ctx, 9, 7, 11, 40, sigma=sigma, tol=1e-12)


def test_odd_axes_take_fewer_iterations(ctx):
    mc = solve_and_compare(ctx, 15, 15, 15, 10)
    assert mc.Iterations.max() <= 60  # the Jacobi loop takes about 290


def test_odd_moved_nodes(ctx):
    """Moved nodes on an odd lattice: the V-cycle of the cube lattice as the preconditioner."""
    n, K, R = 7, 10, 9
    model = M.clamped_block_model(n)
    rng = np.random.default_rng(5)
    inner = (model.xyz > 0.5).all(axis=1) & (model.xyz < n - 0.5).all(axis=1)
    model.xyz[inner] += 0.15 * rng.uniform(-1, 1, (int(inner.sum()), 3))
    kl = M.LognormalStochasticCoefficientsProvider([n, n, n], 0.3 * n, K, 8)
    mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=K, simulations=R, seed=3,
                                                    mode="mixed", tolerance=1e-10)
    mc.Initialize()
    mc.Solve()
    E = O.kl_field(O.centroids(model.xyz, model.conn), [n, n, n], kl.table(), mc.RandomNumbers[:2], sigma=0.3)
    for r in range(2):
        C = O.CSR(model.n_nodes, model.conn, model.dof, model.n_dofs)
        C.assemble(O.h8_stiffness_batch(model.element_xyz(), E[r], model.poisson)[0])
        xo, _ = C.pcg_jacobi(model.subdomains[0].RHS, tol=1e-13)
        assert np.abs(mc.Solutions[r] - xo).max() <= 1e-8 * np.abs(xo).max()
