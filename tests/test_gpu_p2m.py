"""P2M at the node sizes where its work split changes (one source, the lanes' subsets, batches of 32, the
64 sources above which four warps share a node) and orders with every number of order pairs, against
the oracle's multipoles; dipoles against their limit, pairs of opposite charges.

FP64 bar: 1e-13 max-norm relative (the repository's, test/test_device_harmonics.jl's). Dipoles: the
pair of charges ±|d|/h at ±h/2 along d differs from the dipole by (h·n/2)²/6 of the degree-n term and
by the cancellation 2⁻⁵³/h; at h = 1e-4 of the box both stay below 1e-6 of the multipole's largest entry
for n ≤ 14.
"""
import numpy as np
import pytest

from helpers import mrd

pytestmark = pytest.mark.gpu
BOX = ((0.0, 0.0, 0.0), 1.0)


def clumps(rng, sizes):
    """The 64 boxes of a 4 x 4 x 4 grid with the given numbers of points in turn: the nodes of level 2
    (each octant holds more points than the leaf size, none of the boxes does)."""
    pts = []
    for i in range(64):
        o = np.array([i % 4, (i // 4) % 4, i // 16])
        n = sizes[(i + 5 * (i // 16)) % len(sizes)]
        pts.append((o + 0.05 + 0.9 * rng.random((n, 3))) / 4.0)
    return np.concatenate(pts)


SIZES = [1, 2, 3, 5, 16, 31, 32, 33, 63, 64, 65, 96, 97, 128, 200, 300]


@pytest.mark.parametrize("p", [1, 2, 3, 5, 6, 9, 10, 11, 14, 16, 19, 20])
def test_multipoles_match_oracle(oracle, fmmb, p):
    rng = np.random.default_rng(700 + p)
    pts = clumps(rng, SIZES)
    tau = rng.standard_normal(len(pts))
    O = oracle.FMM(p, pts, 300)
    O.build_expansions(pts, tau)
    OM, _ = O.expansions()
    f = fmmb.FMM(fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=p), pts, ppl=300, bbox=BOX)
    M, _ = fmmb.build_expansions(f, pts, tau).expansions()
    assert f.nlevels == 3 and M.shape == OM.shape and mrd(M.ravel(), OM.ravel()) < 1e-13
    if p <= 11:
        Mx, _ = fmmb.build_expansions(f, pts, tau, precision="mixed").expansions()
        # sums of up to 300 FP32 products: 2⁻²⁴ times a few roundings each, 2⁻²⁰ of the sum of magnitudes
        A, _ = fmmb.build_expansions(f, pts, np.abs(tau)).expansions()
        assert np.max(np.abs(Mx - M)) <= 2.0 ** -20 * np.max(np.abs(A))


@pytest.mark.parametrize("p", [1, 2, 4, 8, 14])
def test_dipole_multipoles_match_charge_pairs(fmmb, p):
    rng = np.random.default_rng(720 + p)
    pts = clumps(rng, SIZES)
    n, h = len(pts), 1e-4 * 0.25
    mom = rng.standard_normal((n, 3))
    m = fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=p)
    f = fmmb.FMM(m, pts, ppl=300, bbox=BOX)
    D, _ = fmmb.build_expansions(f, pts, fmmb.Dipoles(mom)).expansions()
    tau = rng.standard_normal(n)
    Q, _ = fmmb.build_expansions(f, pts, tau).expansions()
    B, _ = fmmb.build_expansions(f, pts, (tau, fmmb.Dipoles(mom))).expansions()
    assert mrd(B.ravel(), (D + Q).ravel()) < 1e-13
    e = mom / np.linalg.norm(mom, axis=1)[:, None]
    two = np.concatenate([pts + 0.5 * h * e, pts - 0.5 * h * e])
    q = np.concatenate([np.linalg.norm(mom, axis=1), -np.linalg.norm(mom, axis=1)]) / h
    g = fmmb.FMM(m, two, ppl=600, bbox=BOX)
    assert f.nlevels == 3 and g.nnodes == f.nnodes
    P, _ = fmmb.build_expansions(g, two, q).expansions()
    assert mrd(P.ravel(), D.ravel()) < 1e-6


SMALL = [1, 2, 4, 7, 8, 9, 12, 15, 16, 17]


@pytest.mark.parametrize("p", [1, 2, 3, 4, 7, 8, 12, 15, 16])
def test_small_nodes_match_oracle(oracle, fmmb, p):
    """Nodes of at most 8 and 16 sources, which share a warp up to p = 15."""
    rng = np.random.default_rng(740 + p)
    pts = clumps(rng, SMALL)
    tau = rng.standard_normal(len(pts))
    O = oracle.FMM(p, pts, 20)
    O.build_expansions(pts, tau)
    OM, _ = O.expansions()
    f = fmmb.FMM(fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=p), pts, ppl=20, bbox=BOX)
    M, _ = fmmb.build_expansions(f, pts, tau).expansions()
    assert f.nlevels == 3 and M.shape == OM.shape and mrd(M.ravel(), OM.ravel()) < 1e-13


@pytest.mark.parametrize("p,precision", [(1, "fp64"), (3, "mixed"), (6, "fp64"), (9, "mixed"), (15, "fp64"), (16, "fp64")])
def test_small_nodes_same_in_a_large_launch(fmmb, p, precision):
    """A list that fills the device gives each warp four nodes and each CTA all sets of its nodes (charges and the
    dipoles' components); a node's sums depend on neither: a batch of eight instances, large, equals each
    instance's own plan, small, bit by bit."""
    rng = np.random.default_rng(760 + p)
    m = fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=p)
    sets = [rng.random((30000, 3)) for _ in range(8)]
    tau, mom = [rng.standard_normal(30000) for _ in sets], [0.1 * rng.standard_normal((30000, 3)) for _ in sets]
    batch = fmmb.BatchFMM(m, sets, ppl=24, bbox=BOX)
    cache = fmmb.OperatorCache(m)
    alone = [fmmb.FMM(m, s, ppl=24, bbox=BOX, cache=cache) for s in sets[:2]]
    assert alone[0].nnodes < 8000 and batch.nnodes > 32000
    for dip in (False, True):
        dens = lambda q, d: (q, fmmb.Dipoles(d)) if dip else q
        u = fmmb.evaluate_at_sources(batch, fmmb.build_expansions(batch, batch.sources, dens(batch.concat(tau), np.concatenate(mom)),
                                                                  precision=precision))
        for i, f in enumerate(alone):
            a = fmmb.evaluate_at_sources(f, fmmb.build_expansions(f, sets[i], dens(tau[i], mom[i]), precision=precision))
            assert np.array_equal(batch.split(u)[i], a), (i, dip)
