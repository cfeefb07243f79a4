"""Stress recovery of realization batches at the edges of its work split
(4 elements a warp, 16 a CTA, ranges of realizations), on outputs that start off
a 16-byte boundary, and with values that are not finite. Bound: 1e-12 of each
array's maximum against the oracle (the same FP64 sums, some of them fused), the
bound of the other stress tests."""
import ctypes as C

import numpy as np
import pytest

import msolve_b200 as M
import oracle as O
from msolve_b200 import _native as N

pytestmark = pytest.mark.gpu


def recover(ctx, model, E, X, offset):
    import torch
    dev = torch.device("cuda")
    R, ne = E.shape
    mesh = M.GpuMesh(ctx, model)
    bufs = [torch.zeros(R * ne * k + 1, dtype=torch.float64, device=dev) for k in (48, 48, 24)]
    e, x = torch.from_numpy(E).to(dev), torch.from_numpy(X).to(dev)
    torch.cuda.synchronize()
    N.check(N.lib().MSG_STRESS_BATCH_DEVICE(mesh.handle, R, C.c_void_p(e.data_ptr()), 0.3, C.c_void_p(x.data_ptr()),
                                            *(C.c_void_p(b.data_ptr() + 8 * offset) for b in bufs)), ctx.handle)
    out = [b.cpu().numpy()[offset:offset + R * ne * k] for b, k in zip(bufs, (48, 48, 24))]
    return [o.reshape(R, ne, -1) for o in out]


def oracle(model, E, X):
    out = [[], [], []]
    xyz = model.element_xyz()
    for r in range(E.shape[0]):
        full = np.zeros((model.n_nodes, 3))
        full[model.dof >= 0] = X[r][model.dof[model.dof >= 0]]
        u = full[model.conn].reshape(-1, 24)
        eps, sig, f, st = O.h8_stress_batch(xyz, E[r], 0.3, u)
        assert st == 0
        for o, v in zip(out, (eps, sig, f)):
            o.append(np.asarray(v).reshape(model.n_elems, -1))
    return [np.array(o) for o in out]


@pytest.mark.parametrize("nx,ny,nz,R,offset", [(1, 1, 1, 1, 0), (3, 1, 1, 2, 1), (2, 2, 1, 65, 0), (5, 1, 1, 3, 1),
                                               (4, 2, 2, 7, 0), (17, 1, 1, 9, 1), (5, 4, 3, 33, 0)])
def test_batch_edges(ctx, nx, ny, nz, R, offset):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    rng = np.random.default_rng(nx + R)
    model.xyz += 0.1 * rng.uniform(-1, 1, model.xyz.shape)
    E = rng.uniform(0.5, 2.0, (R, model.n_elems))
    X = 0.01 * rng.standard_normal((R, model.n_dofs))
    for got, want in zip(recover(ctx, model, E, X, offset), oracle(model, E, X)):
        assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_values_that_are_not_finite(ctx, bad):
    """The products with the zeros of B and D count: the same entries are NaN as
    with the full matrix products."""
    model = M.clamped_block_model(3, ny=2, nz=2)
    rng = np.random.default_rng(1)
    E = rng.uniform(0.5, 2.0, (3, model.n_elems))
    X = 0.01 * rng.standard_normal((3, model.n_dofs))
    X[1, 4] = bad
    E[2, 5] = bad
    for got, want in zip(recover(ctx, model, E, X, 0), oracle(model, E, X)):
        fine = np.isfinite(want)
        assert np.array_equal(fine, np.isfinite(got)) and np.array_equal(np.isnan(want), np.isnan(got))
        assert np.abs(got[fine] - want[fine]).max() <= 1e-12 * np.abs(want[fine]).max()


def test_stresses_that_overflow(ctx):
    """Finite strains and moduli whose product is not: a stretch along x of 1e300 at a
    modulus of 1e10 (its rounding in the other strains, 1e284, stays finite there). The
    force of every node is then NaN, the sum of products of infinite stresses with the
    zeros of B."""
    model = M.clamped_block_model(3, ny=2, nz=2)
    rng = np.random.default_rng(1)
    E = rng.uniform(0.5, 2.0, (3, model.n_elems))
    X = 0.01 * rng.standard_normal((3, model.n_dofs))
    E[1] = 1e10
    X[1] = 0.0
    free = model.dof[:, 0] >= 0
    X[1, model.dof[free, 0]] = 1e300 * model.xyz[free, 0]
    for got, want in zip(recover(ctx, model, E, X, 0), oracle(model, E, X)):
        assert np.array_equal(np.isfinite(want), np.isfinite(got)) and np.array_equal(np.isnan(want), np.isnan(got))
    assert np.isnan(want[1]).all()
