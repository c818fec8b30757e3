"""The radix sort behind the tree, on both sides of the size where its tiles change (148 tiles of 4,096
keys): every leaf's points lie in its cell, in their original order, and each point in one leaf."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOX = ((0.0, 0.0, 0.0), 1.0)


@pytest.mark.parametrize("n", [1, 255, 1025, 148 * 4096 - 1, 148 * 4096])
def test_points_sorted_by_leaf(fmmb, n):
    x = np.random.default_rng(n).random((n, 3))
    f = fmmb.FMM(fmmb.SphericalHarmonics(fmmb.Laplace3D(), p=2), x, ppl=100, bbox=BOX)
    t = f.tree()
    perm = t["perm"]
    assert np.array_equal(np.sort(perm), np.arange(n))
    leaf = np.nonzero((t["child_first"] < 0) & t["has_source"].astype(bool))[0]
    lo, cnt = t["plo"][leaf], t["phi"][leaf] - t["plo"][leaf] + 1
    order = np.argsort(lo)
    leaf, lo, cnt = leaf[order], lo[order], cnt[order]
    assert np.array_equal(lo, np.concatenate([[0], np.cumsum(cnt)[:-1]])) and cnt.sum() == n
    of = np.repeat(np.arange(len(leaf)), cnt)
    same = of[1:] == of[:-1]
    assert np.all(perm[1:][same] > perm[:-1][same])
    w = 0.5 ** t["level"][leaf][of]
    lower = t["cell"][leaf][of][:, :3] * w[:, None]
    assert np.all(x[perm] >= lower) and np.all(x[perm] <= lower + w[:, None])
