"""The FP64 M2L by rotations against the oracle's dense class operators, at the orders where its
blocks change shape (p + 1 below, at and above 4, 8, 12, 16 and 20, and the launch's own limits) and
on trees with full chunks (uniform), ragged ones (a sphere) and a few pairs per class (a small tree).

The bar is the repository's FP64 one (1e-12 and 1e-11 max-norm relative on potentials and
gradients): the factored translation is exact, so the two differ by rounding, a few units in 1e-16
per factor of the blocks' norms.
"""
import numpy as np
import pytest

from helpers import DISTRIBUTIONS3, mrd

pytestmark = pytest.mark.gpu
BOX = ((0.0, 0.0, 0.0), 1.0)


@pytest.mark.parametrize("p", [1, 2, 3, 4, 6, 7, 8, 11, 12, 13, 15, 16, 17, 18, 19, 20])
def test_rotated_m2l_matches_dense(oracle, fmmb, p):
    for name, n, ppl in (("uniform", 2500, 20), ("sphere", 2000, 25), ("clustered", 700, 30)):
        rng = np.random.default_rng(90 + p)
        pts = DISTRIBUTIONS3[name](rng, n)
        tau = rng.standard_normal(n)
        O = oracle.FMM(p, pts, ppl)
        O.build_expansions(pts, tau)
        ou, og = O.evaluate_at_sources()
        f = fmmb.FMM(fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=p), pts, ppl=ppl, bbox=BOX)
        u, g = fmmb.evaluate_at_sources_both(f, fmmb.build_expansions(f, pts, tau))
        assert mrd(u, ou) < 1e-12 and mrd(g, og) < 1e-11, (name, mrd(u, ou), mrd(g, og))


def test_order_16_same_in_a_large_launch(fmmb):
    """At p = 16 a launch of 600,000 pairs or more takes another shape (two groups of warps, chunks of
    24 pairs). A pair's product and the order of a target's sums depend on neither: a batch of eight
    instances, large, equals each instance's own plan, small, bit by bit."""
    rng = np.random.default_rng(16)
    m = fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=16)
    sets = [DISTRIBUTIONS3["uniform"](rng, 6000) for _ in range(8)]
    tau = [rng.standard_normal(6000) for _ in sets]
    batch = fmmb.BatchFMM(m, sets, ppl=4, bbox=BOX)
    cache = fmmb.OperatorCache(m)
    alone = [fmmb.FMM(m, s, ppl=4, bbox=BOX, cache=cache) for s in sets]
    assert max(f.npairs for f in alone) < 600000 <= batch.npairs
    u, g = fmmb.evaluate_at_sources_both(batch, fmmb.build_expansions(batch, batch.sources, batch.concat(tau)))
    for i, f in enumerate(alone):
        a, b = fmmb.evaluate_at_sources_both(f, fmmb.build_expansions(f, sets[i], tau[i]))
        assert np.array_equal(batch.split(u)[i], a) and np.array_equal(batch.split(g)[i], b)


@pytest.mark.parametrize("p", [4, 8, 11, 14, 20])
def test_same_bits_whatever_the_parts(fmmb, p):
    """A skewed tree's blocks are cut into more parts than a uniform one's (the heaviest block decides): an instance
    of a batch whose other instance is one dense cluster equals its own plan bit by bit."""
    rng = np.random.default_rng(50 + p)
    m = fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=p)
    sets = [rng.random((3000, 3)), np.clip(0.5 + 0.02 * rng.standard_normal((20000, 3)), 0.0, 1.0)]
    tau = [rng.standard_normal(len(s)) for s in sets]
    batch = fmmb.BatchFMM(m, sets, ppl=16, bbox=BOX)
    cache = fmmb.OperatorCache(m)
    u, g = fmmb.evaluate_at_sources_both(batch, fmmb.build_expansions(batch, batch.sources, batch.concat(tau)))
    for i, s in enumerate(sets):
        f = fmmb.FMM(m, s, ppl=16, bbox=BOX, cache=cache)
        a, b = fmmb.evaluate_at_sources_both(f, fmmb.build_expansions(f, s, tau[i]))
        assert np.array_equal(batch.split(u)[i], a) and np.array_equal(batch.split(g)[i], b)
