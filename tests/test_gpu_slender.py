"""Batched mixed solves on slender lattices, columns and slabs, cubes and moved nodes:
they converge, the lattices in no more iterations than in the Jacobi loop (option
multigrid = 0; on such moved meshes that loop itself runs into its limit). The
residual of the returned displacements, formed here from the element matrices, stays
below the tolerance plus its own rounding: a row of K x is a sum of some 200 products
(8 elements of 24), and numpy's FP64 sums of them lose at most 200 units of the
rounding of |K| |x|."""
import numpy as np
import pytest

import msolve_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu
TERMS, TOL = 50, 1e-10


def residual(model, E, x):
    """||b - K x|| / ||b|| and its rounding."""
    Ke = O.unpack300(O.h8_stiffness_batch(model.element_xyz(), E, model.poisson)[0])
    full = np.zeros((model.n_nodes, 3))
    free = model.dof >= 0
    full[free] = x[model.dof[free]]
    u = full[model.conn].reshape(-1, 24)

    def assembled(K, v):
        y = np.zeros((model.n_nodes, 3))
        np.add.at(y, model.conn.reshape(-1), np.einsum("eij,ej->ei", K, v).reshape(-1, 3))
        out = np.zeros(model.n_dofs)
        out[model.dof[free]] = y[free]
        return out

    b = model.subdomains[0].RHS
    bound = 200 * np.finfo(float).eps * np.linalg.norm(assembled(np.abs(Ke), np.abs(u)))
    return np.linalg.norm(b - assembled(Ke, u)) / np.linalg.norm(b), bound / np.linalg.norm(b)


def solve(ctx, model, kl, xi):
    mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=TERMS, simulations=len(xi),
                                                    mode="mixed", tolerance=TOL)
    mc.RandomNumbers = xi
    mc.Solve()  # (raises when a realization does not converge)
    return mc


@pytest.mark.parametrize("nx,ny,nz,R,moved", [(5, 5, 90, 1, False), (5, 5, 90, 16, False), (7, 7, 90, 4, False),
                                              (7, 9, 64, 1, False), (5, 9, 64, 1, False), (3, 3, 40, 1, False),
                                              (4, 5, 64, 16, False), (6, 10, 60, 1, False), (6, 52, 52, 1, False),
                                              (5, 5, 90, 2, True), (3, 3, 40, 2, True)])
def test_slender(ctx, nx, ny, nz, R, moved):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    if moved:
        rng = np.random.default_rng(7)
        inner = (model.xyz > 0.5).all(axis=1) & (model.xyz < np.array([nx, ny, nz]) - 0.5).all(axis=1)
        model.xyz[inner] += 0.15 * rng.uniform(-1, 1, (int(inner.sum()), 3))
    sides = [nx, ny, nz]
    kl = M.LognormalStochasticCoefficientsProvider(sides, 0.2 * nx, TERMS, 16)
    xi = np.random.default_rng(1).standard_normal((R, TERMS))
    mc = solve(ctx, model, kl, xi)
    if not moved:
        ctx.set_option("multigrid", 0)
        try:
            jacobi = solve(ctx, model, kl, xi)
        finally:
            ctx.set_option("multigrid", 1)
        assert mc.Iterations.max() <= jacobi.Iterations.max()
    E = O.kl_field(O.centroids(model.xyz, model.conn), sides, kl.table(), xi, sigma=kl.sigma)
    for r in (0, R - 1):
        rel, rounding = residual(model, E[r], mc.Solutions[r])
        assert rel <= TOL + rounding, (r, rel, rounding)
