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


def few_and_many(ctx, solve, few, many):
    """Results of the first `few` realizations alone and within `many`."""
    ctx.set_option("fixed_updates", 1)  # a realization's updates do not depend on the others
    try:
        return solve(few), solve(many)
    finally:
        ctx.set_option("fixed_updates", 0)


# long axes are walked in segments by small batches, whole by large ones: partial
# sums per chunk of planes, so that the same numbers come out to the last bit. Axes
# of 6 to 40 elements: chunks of 3 to 10 planes, the last one short or of one plane
@pytest.mark.parametrize("nx,ny,nz,many", [(6, 6, 6, 300), (12, 12, 12, 1000), (13, 10, 7, 900), (25, 4, 4, 1100),
                                           (40, 5, 5, 700)])
def test_segments_give_the_same_numbers(ctx, nx, ny, nz, many):
    few, K = 2, 12
    xi = np.random.default_rng(nx).standard_normal((many, K))
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    kl = M.LognormalStochasticCoefficientsProvider([nx, ny, nz], 0.3 * nx, K, 8)

    def solve(R):
        mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=K, simulations=R, seed=1,
                                                        mode="mixed", tolerance=1e-10)
        mc.Initialize()
        mc.RandomNumbers = xi[:R]
        mc.Solve()
        return mc.Solutions[:few].copy(), mc.Iterations[:few].copy()

    (xf, itf), (xm, itm) = few_and_many(ctx, solve, few, many)
    assert np.array_equal(itf, itm)
    assert np.array_equal(xf, xm)


@pytest.mark.parametrize("n,R", [(5, 2), (9, 3), (10, 17)])
def test_newmark_segments(ctx, n, R):
    """The Jacobi loop in segments against the oracle's direct solves, with the
    bounds of the batched Newmark parity test (tip 1e-8, final field 1e-7: each
    step is solved to 1e-11)."""
    steps, dt = 6, 0.01
    model = M.clamped_block_model(n)
    kl = M.LognormalStochasticCoefficientsProvider([n, n, n], 0.2 * n, 12, 6)
    load = M.MassAccelerationSinusoidalLoad(1.0, dt, dt * steps, 0.1, dof=0)
    corner = int(np.argmax(model.xyz.sum(1)))
    nm = M.NewmarkDynamicAnalyzer(ctx, model, kl, 0.25, 0.5, dt, dt * steps, load, expansion_order=12,
                                  simulations=R, density=1.0, rayleigh_alpha=0.01, rayleigh_beta=0.001,
                                  tolerance=1e-11, tip_dof=int(model.dof[corner, 0]))
    nm.RandomNumbers = np.random.default_rng(n).standard_normal((R, 12))
    hist = nm.Solve()
    E = O.kl_field(O.centroids(model.xyz, model.conn), [n, n, n], kl.table(), nm.RandomNumbers, mean=kl.mean,
                   sigma=kl.sigma, mean_correction=kl.mean_correction)
    cons = (model.dof < 0).astype(np.uint8)
    for r in (0, R - 1):
        t, u, info = O.block_newmark(n, n, n, cons, E[r], model.poisson, 1.0, 0.01, 0.001, 0.25, 0.5, dt, steps, 0.1,
                                     1.0, 0, model.n_dofs, tip_dof=nm.tip_dof)
        assert info["status"] == 0
        assert np.abs(hist[r] - t).max() <= 1e-8 * np.abs(t).max()
        assert np.abs(nm.Solutions[r] - u).max() <= 1e-7 * np.abs(u).max()


# moved nodes: node counts around the element-by-element work items (8 and 32
# nodes), the last one short; by the diagonal (under 216 elements on odd axes) and by
# the V-cycle; one to four realization groups
@pytest.mark.parametrize("nx,ny,nz,R", [(1, 1, 1, 3), (3, 3, 3, 33), (3, 1, 2, 40), (4, 4, 4, 64), (6, 5, 8, 100)])
def test_moved_node_counts(ctx, nx, ny, nz, R):
    K = 6
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    rng = np.random.default_rng(R)
    top = np.array([nx, ny, nz])
    free = (model.xyz > 0.5).all(axis=1) | (model.xyz == top).any(axis=1)
    model.xyz[free] += 0.1 * rng.uniform(-1, 1, (int(free.sum()), 3))
    kl = M.LognormalStochasticCoefficientsProvider([nx, ny, nz], 0.3 * nx, K, 8)
    mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=K, simulations=R, seed=3,
                                                    mode="mixed", tolerance=1e-10)
    mc.Initialize()
    mc.Solve()
    rows = (0, R - 1)
    E = O.kl_field(O.centroids(model.xyz, model.conn), [nx, ny, nz], kl.table(), mc.RandomNumbers[list(rows)], sigma=0.3)
    for i, r in enumerate(rows):
        C = O.CSR(model.n_nodes, model.conn, model.dof, model.n_dofs)
        C.assemble(O.h8_stiffness_batch(model.element_xyz(), E[i], model.poisson)[0])
        xo, _ = C.pcg_jacobi(model.subdomains[0].RHS, tol=1e-13)
        assert np.abs(mc.Solutions[r] - xo).max() <= 1e-8 * np.abs(xo).max()


# all sweeps of the coarsest level in one launch against a launch a sweep, bit for
# bit: 8 realizations a CTA, the last one short; coarsest levels with fewer nodes than
# a CTA's lanes take at a time, and with several rounds of them
@pytest.mark.parametrize("nx,ny,nz,R", [(6, 6, 6, 1), (4, 4, 4, 9), (40, 5, 5, 17), (10, 30, 26, 5)])
def test_fused_coarsest_sweeps(ctx, nx, ny, nz, R):
    model = M.clamped_block_model(nx, ny=ny, nz=nz)
    kl = M.LognormalStochasticCoefficientsProvider([nx, ny, nz], 0.3 * nx, 8, 8)
    out = []
    for fused in (0, 1):
        ctx.set_option("multigrid_fused_coarse", fused)
        try:
            mc = M.MonteCarloAnalyzerWithStochasticMaterial(ctx, model, kl, expansion_order=8, simulations=R, seed=2,
                                                            mode="mixed", tolerance=1e-10)
            mc.Initialize()
            mc.Solve()
        finally:
            ctx.set_option("multigrid_fused_coarse", 1)
        out.append((mc.Solutions.copy(), mc.Iterations.copy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
