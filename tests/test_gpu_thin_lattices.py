"""Thin lattices with an odd side on which a V-cycle costs more than the iterations it
saves keep to the Jacobi loop: the iterations and bits of option multigrid = 0. Slabs
and columns three and four elements thick, and the largest small one."""
import numpy as np
import pytest

import msolve_b200 as M

pytestmark = pytest.mark.gpu
TERMS = 20


@pytest.mark.parametrize("nx,ny,nz,R", [(40, 40, 3, 2), (3, 40, 40, 1), (3, 30, 24, 17), (12, 12, 3, 1), (3, 3, 40, 2),
                                        (17, 17, 4, 1), (5, 5, 5, 3), (41, 41, 4, 1)])
def test_keeps_to_the_jacobi_loop(ctx, nx, ny, nz, R):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    kl = M.LognormalStochasticCoefficientsProvider([nx, ny, nz], 0.2 * nx, TERMS, 10)
    out = []
    for multigrid in (1, 0):
        ctx.set_option("multigrid", multigrid)
        try:
            mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=TERMS, simulations=R, seed=4,
                                                            mode="mixed", tolerance=1e-10)
            mc.Initialize()
            mc.Solve()
        finally:
            ctx.set_option("multigrid", 1)
        out.append(mc)
    assert np.array_equal(out[0].Iterations, out[1].Iterations)
    assert np.array_equal(out[0].Solutions, out[1].Solutions)
