"""The near field's frame at the sizes where it changes: targets per chunk (lane splits at 4, 8, 16,
chunks of 32, pairs of chunks of 64) and the pairs above which a team of warps takes the leaf
(10,000: 100 targets of 100 sources), on trees of one leaf, whose evaluation is the near field alone.

FP64 bars: 1e-13 max-norm relative (the repository's bar for a single leaf: sums of up to 300 terms in
FP64, a few units in 1e-16 each). FP32: each term carries a few roundings of 2⁻²⁴ (differences, square
norm, reciprocal root below 2⁻²², products) and batches of 32 are summed in FP32, so the error stays
below 2⁻¹⁹ of the sum of the terms' magnitudes.
"""
import numpy as np
import pytest

from helpers import mrd, stokes_direct

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 36, 40, 48, 49, 63, 64, 65, 96, 97, 100, 101, 128, 129, 160, 200, 300]
BOX = ((0.0, 0.0, 0.0), 1.0)


@pytest.mark.parametrize("n", SIZES)
def test_one_leaf_equals_direct(oracle, fmmb, n):
    rng = np.random.default_rng(1000 + n)
    pts, tau = rng.random((n, 3)), rng.standard_normal(n)
    tg = rng.random((n // 2 + 1, 3))
    du, dg = oracle.direct(pts, tau)
    m = fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=4)
    f = fmmb.FMM(m, pts, ppl=300, bbox=BOX)
    st = fmmb.build_expansions(f, pts, tau)
    u, g = fmmb.evaluate_at_sources_both(f, st)
    assert np.array_equal(u, fmmb.evaluate_at_sources(f, st))          # with and without the gradient
    d = tg[:, None, :] - pts[None, :, :]
    r = np.sqrt((d * d).sum(-1))
    tu = (tau / r).sum(1) / (4 * np.pi)
    assert mrd(fmmb.evaluate(f, st, tg), tu) < 1e-13
    d = pts[:, None, :] - pts[None, :, :]
    r = np.sqrt((d * d).sum(-1))
    np.fill_diagonal(r, np.inf)
    mom = rng.standard_normal((n, 3))
    dd = np.einsum("tsk,sk->ts", d, mom)
    sd = fmmb.build_expansions(f, pts, (tau, fmmb.Dipoles(mom)))
    ref = du + (dd / r ** 3).sum(1) / (4 * np.pi)
    y = fmmb.FMM(fmmb.SphericalHarmonics(fmmb.Yukawa3D(5.0), p=4), pts, ppl=300, bbox=BOX)
    yu, yg = fmmb.evaluate_at_sources_both(y, fmmb.build_expansions(y, pts, tau))
    e = np.where(np.isinf(r), 0.0, np.exp(-5.0 * np.where(np.isinf(r), 0.0, r)) / r) * tau
    eu = e.sum(1) / (4 * np.pi)
    eg = -np.einsum("ts,tsk->tk", e * np.where(np.isinf(r), 0.0, 1 + 5.0 * np.where(np.isinf(r), 0.0, r)) / r ** 2, d) / (4 * np.pi)
    sp = fmmb.StokesFMMPlan(pts, p=4, ppl=300, bbox=BOX)
    v = fmmb.stokes_fmm_eval(sp, stokeslets=mom)
    mx = fmmb.build_expansions(f, pts, tau, precision="mixed")
    fu, fg = fmmb.evaluate_at_sources_both(f, mx)
    if n == 1:
        for a in (u, g, yu, yg, v, fu, fg, fmmb.evaluate_at_sources(f, sd)):
            assert np.all(a == 0)
        return
    assert mrd(u, du) < 1e-13 and mrd(g, dg) < 1e-13
    assert mrd(fmmb.evaluate_at_sources(f, sd), ref) < 1e-13
    assert mrd(yu, eu) < 1e-13 and mrd(yg, eg) < 1e-13
    assert mrd(v, stokes_direct(pts, mom, np.arange(n))) < 1e-13
    size = (np.abs(tau) / r).sum(1) / (4 * np.pi)
    gsize = (np.abs(tau) / r ** 2).sum(1) / (4 * np.pi)
    assert np.all(np.abs(fu - du) <= 2.0 ** -19 * size)
    assert np.all(np.linalg.norm(fg - dg, axis=1) <= 2.0 ** -19 * gsize)


def test_coincident_points(fmmb):
    """Two sources at one place: their potentials are infinite on the FP64 path, and nobody else's is."""
    rng = np.random.default_rng(5)
    pts, tau = rng.random((150, 3)), np.abs(rng.standard_normal(150)) + 0.1
    pts[7] = pts[90]
    f = fmmb.FMM(fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=4), pts, ppl=300, bbox=BOX)
    u = fmmb.evaluate_at_sources(f, fmmb.build_expansions(f, pts, tau))
    assert np.isposinf(u[[7, 90]]).all() and np.isfinite(np.delete(u, [7, 90])).all()
