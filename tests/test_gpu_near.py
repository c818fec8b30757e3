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

from helpers import mrd, stokes_direct, stokes_direct_all

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


SPLITS = [1, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 100, 101, 200]


@pytest.mark.parametrize("n", SPLITS)
@pytest.mark.parametrize("output", ["velocity", "pressure", "gradient"])
def test_one_leaf_stokes_densities(fmmb, n, output):
    """Every Stokes density and output at the sources, and at fewer and more targets than sources: chunks of 32
    (densities, gradients) and of 64 (Stokeslets). Bar: as above, sums of a dozen products a source."""
    rng = np.random.default_rng(2000 + n)
    pts, z = rng.random((n, 3)), lambda: rng.standard_normal((n, 3))
    d = dict(stokeslets=z(), stresslets=z(), stressvecs=z(), doublets=z())
    one = dict(stokeslets=d["stokeslets"])
    p = fmmb.StokesFMMPlan(pts, p=4, ppl=300, bbox=BOX)
    tg = [rng.random((m, 3)) for m in (1, max(1, n // 2), 130)]
    for dens in (d, one):
        r = dict(f=dens["stokeslets"], fs=dens.get("stresslets"), nu=dens.get("stressvecs"), g=dens.get("doublets"))
        want = stokes_direct_all(pts, np.arange(n), output=output, **r)
        got = fmmb.stokes_fmm_eval(p, output=output, **dens)
        if n == 1:
            assert np.all(got == 0)
        else:
            assert np.max(np.abs(got - want)) < 1e-13 * np.max(np.abs(want))
        for t in tg:
            want = stokes_direct_all(pts, None, output=output, tgt=t, **r)
            got = fmmb.stokes_fmm_eval(p, output=output, targets=t, **dens)
            assert np.max(np.abs(got - want)) < 1e-13 * np.max(np.abs(want))


@pytest.mark.parametrize("n", SPLITS)
def test_one_leaf_mixed_targets_and_dipoles(fmmb, n):
    """The mixed path's targets, and its dipoles at sources and targets. Bar: 2⁻¹⁹ of the sum of the terms'
    magnitudes for their roundings, as above, and their change under the rounding of the positions: leaf-centred
    coordinates below ½ are rounded by at most 2⁻²⁶, a difference by 2⁻²⁵, a distance vector by √3·2⁻²⁵, times the
    terms' derivatives (1/r² and 4/r³ of a charge's potential and gradient, 4/r³ and 24/r⁴ of a dipole's).
    """
    rng = np.random.default_rng(3000 + n)
    pts, tau, mom = rng.random((n, 3)), rng.standard_normal(n), rng.standard_normal((n, 3))
    f = fmmb.FMM(fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=4), pts, ppl=300, bbox=BOX)
    for dip in (False, True):
        st = fmmb.build_expansions(f, pts, (tau, fmmb.Dipoles(mom)) if dip else tau, precision="mixed")
        for t in (pts, rng.random((1, 3)), rng.random((max(1, n // 2), 3)), rng.random((130, 3))):
            v = t[:, None, :] - pts[None, :, :]
            r = np.sqrt((v * v).sum(-1))
            if t is pts:
                np.fill_diagonal(r, np.inf)
                u = fmmb.evaluate_at_sources(f, st)
                g = fmmb.evaluate_at_sources(f, st, output=fmmb.Gradient())
            else:
                u, g = fmmb.evaluate(f, st, t), fmmb.evaluate(f, st, t, output=fmmb.Gradient())
            dv = np.einsum("tsk,sk->ts", v, mom) if dip else np.zeros_like(r)
            dm, m1 = (mom, np.linalg.norm(mom, axis=1)) if dip else (np.zeros_like(mom), np.zeros(n))
            ou = (tau / r + dv / r ** 3).sum(1) / (4 * np.pi)
            og = (np.einsum("ts,sk->tk", 1 / r ** 3, dm) - np.einsum("ts,tsk->tk", tau / r ** 3 + 3 * dv / r ** 5, v)) / (4 * np.pi)
            size = (np.abs(tau) / r + m1 / r ** 2).sum(1) / (4 * np.pi)
            gsize = (np.abs(tau) / r ** 2 + 4 * m1 / r ** 3).sum(1) / (4 * np.pi)
            shift = 3 ** 0.5 * 2.0 ** -25 / (4 * np.pi)
            moved = shift * (np.abs(tau) / r ** 2 + 4 * m1 / r ** 3).sum(1)
            gmoved = shift * (4 * np.abs(tau) / r ** 3 + 24 * m1 / r ** 4).sum(1)
            assert np.all(np.abs(u - ou) <= 2.0 ** -19 * size + moved)
            assert np.all(np.linalg.norm(g - og, axis=1) <= 2.0 ** -19 * gsize + gmoved)
