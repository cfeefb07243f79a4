"""Batches of different sizes one after another on one mesh and context, whose
buffers and work items agree and whose loop graph is therefore kept: the larger
batch that follows a smaller one takes the iterations and gives the bits that it
gives on a context of its own. Update schedule fixed, so that a realization's steps
do not depend on the others. Sizes: the smaller and the larger batch fill the same
16-wide realization groups (an even number of them from five on) but other numbers
of the coarsest level's 8-wide ones."""
import numpy as np
import pytest

import msolve_b200 as M

pytestmark = pytest.mark.gpu
TERMS = 10


def germs(n, R):
    return np.random.default_rng(n).standard_normal((R, TERMS))


def model_and_field(n):
    return M.clamped_block_model(n), M.LognormalStochasticCoefficientsProvider([n] * 3, 0.3 * n, TERMS, 8)


def fixed_context():
    c = M.Context(0)
    c.set_option("fixed_updates", 1)
    return c


@pytest.mark.parametrize("n,few,many", [(8, 1, 9), (8, 33, 48), (6, 65, 96), (7, 3, 16)])
def test_larger_batch_after_a_smaller_one(n, few, many):
    model, kl = model_and_field(n)
    xi = germs(n, many)

    def solves(sizes):
        mc = M.MonteCarloAnalyzerWithStochasticMaterial(fixed_context(), model, kl, expansion_order=TERMS,
                                                        simulations=many, mode="mixed", tolerance=1e-10)
        for R in sizes:
            mc.simulations, mc.RandomNumbers = R, xi
            mc.Solve()
        return mc.Solutions, mc.Iterations

    x, its = solves([few, many])
    x1, its1 = solves([many])
    assert np.array_equal(its, its1)
    assert np.array_equal(x, x1)


@pytest.mark.parametrize("few,many", [(2, 12), (66, 95)])
def test_larger_lattice_batch_of_a_ragged_call(few, many):
    """The same for the cube lattices of a ragged batch, which step side by side."""
    sides = (6, 8)

    def solves(sizes):
        batch = M.RaggedMonteCarloBatch(fixed_context(), tolerance=1e-10)
        for n in sides:
            batch.add(*model_and_field(n), germs(n, many))
        for R in sizes:
            for n, y in zip(sides, batch.systems):
                y["xi"] = np.ascontiguousarray(germs(n, many)[:R])
            results = batch.Solve()
        return results

    for r, r1 in zip(solves([few, many]), solves([many])):
        assert np.array_equal(r["Iterations"], r1["Iterations"])
        assert np.array_equal(r["Solutions"], r1["Solutions"])
