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
