"""The Galerkin product at the edges of its node tiles (8 x 4 x 4) and on bases of
one degree and of repeated terms per matrix, against the oracle. Bound: 1e-12 of
the maximum (the same FP64 products in another order), as tests/test_gpu_pc.py."""
import numpy as np
import pytest

import msolve_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,m,p", [(1, 1, 1, 2, 1), (7, 3, 3, 2, 2), (8, 4, 4, 1, 3), (9, 2, 5, 3, 1),
                                          (16, 7, 8, 2, 2)])
def test_tile_edges(ctx, nx, ny, nz, m, p):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    L = [nx, ny, nz]
    kl = M.GaussianStochasticCoefficientsProvider(L, 0.3 * nx, max(m, 4), 8, mean=1.5, covariance=0.2)
    op = M.PolynomialChaosSolverPCGMatrixCalculator(M.GpuMesh(ctx, model), kl, m, p)
    u = np.random.default_rng(nx + m).standard_normal((op.PsiSize, model.n_dofs))
    y = op.MultiplyWithMatrix(u)
    cen = O.centroids(model.xyz, model.conn)
    csr = O.CSR(model.n_nodes, model.conn, model.dof, model.n_dofs)
    vals = []
    for i in range(m + 1):
        unit = np.zeros((1, kl.n_terms))
        if i:
            unit[0, i - 1] = 1.0
        E = O.kl_field_gaussian(cen, L, kl.table(), unit, kl.mean, kl.covariance)[0] - (kl.mean if i else 0.0)
        csr.assemble(O.h8_stiffness_batch(model.element_xyz(), E, model.poisson)[0])
        vals.append(csr.val.copy())
    yo = O.pc_gaussian_matvec(csr, np.array(vals), m, p, u)
    assert np.abs(y - yo).max() <= 1e-12 * np.abs(yo).max()
    assert np.array_equal(y, op.MultiplyWithMatrix(u))  # the kept buffers change nothing
