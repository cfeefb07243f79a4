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


def solve_and_compare(ctx, nx, ny, nz, R, K=12):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    L = [nx, ny, nz]
    kl = M.LognormalStochasticCoefficientsProvider(L, 0.3 * nx, K, 8)
    mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=K, simulations=R, seed=nx + ny + nz,
                                                    mode="mixed", tolerance=1e-10)
    mc.Initialize()
    mc.Solve()
    rows = sorted({0, R // 2, R - 1})
    E = O.kl_field(O.centroids(model.xyz, model.conn), L, kl.table(), mc.RandomNumbers[rows], sigma=0.3)
    cons = (model.dof < 0).astype(np.uint8)
    for i, r in enumerate(rows):
        xo, _ = O.block_solve_pcg(nx, ny, nz, cons, E[i], model.poisson, model.subdomains[0].RHS, tol=1e-13)
        assert np.abs(mc.Solutions[r] - xo).max() <= 1e-8 * np.abs(xo).max(), (r, nx, ny, nz)
    return mc


# nodes across a tile of 7 x 3 node pencils: one short, exact, one more, in y and z
@pytest.mark.parametrize("nx,ny,nz,R", [(4, 4, 4, 3), (6, 6, 4, 17), (4, 8, 8, 64), (8, 12, 6, 65), (10, 14, 10, 16)])
def test_tile_edges(ctx, nx, ny, nz, R):
    solve_and_compare(ctx, nx, ny, nz, R)
