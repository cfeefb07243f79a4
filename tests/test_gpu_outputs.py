"""Large outputs copied to the host by several threads (8 MB and more of pageable
memory in one call) hold the bits of the same outputs copied plainly: the field of
many realizations against that of parts of them, pageable and pinned, with lengths
that are not whole copy pieces."""
import ctypes as C

import numpy as np
import pytest

import msolve_b200 as M
from msolve_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [607, 700, 1201])
def test_large_outputs(ctx, R):
    torch = pytest.importorskip("torch")
    n, K = 12, 5
    mesh = M.GpuMesh(ctx, M.clamped_block_model(n))
    kl = M.LognormalStochasticCoefficientsProvider([n] * 3, 0.3 * n, K, 6)
    xi = np.random.default_rng(R).standard_normal((R, K))
    E = kl.field(mesh, xi)  # 1,728 doubles a realization
    parts = np.concatenate([kl.field(mesh, xi[i:i + 200]) for i in range(0, R, 200)])
    assert np.array_equal(E, parts)
    pinned = torch.empty((R, n ** 3), dtype=torch.float64, pin_memory=True)
    s = kl.struct()
    N.check(N.lib().MSG_KL_FIELD(mesh.handle, C.byref(s), R, N.ptr(xi), C.cast(pinned.data_ptr(), N._d)), ctx.handle)
    assert np.array_equal(pinned.numpy(), parts)
