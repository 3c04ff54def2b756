"""Member sums and unit rows at the widths and counts their kernels change at,
against the same sums in numpy float32 / float64, one after the other."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


def lloyd_step(x, cent, spherical):
    """One Lloyd iteration in the library's arithmetic: nearest by exact float64
    distance (the rows here are far from ties), member sums in point order in
    float32, means, and for spherical k-means unit length by a float64 norm."""
    d2 = ((x[:, None, :].astype(np.float64) - cent[None].astype(np.float64)) ** 2).sum(2)
    lab = d2.argmin(1)
    out = np.zeros_like(cent)
    for c in range(len(cent)):
        s = np.zeros(x.shape[1], np.float32)
        for row in x[lab == c]:
            s = (s + row).astype(np.float32)
        n = int((lab == c).sum())
        assert n > 0
        m = (s / np.float32(n)).astype(np.float32)
        if spherical:
            sq = np.float64(0.0)
            for v in m.astype(np.float64):
                sq = sq + v * v
            m = (m * np.float32(1.0 / np.sqrt(sq))).astype(np.float32)
        out[c] = m
    return out


@pytest.mark.parametrize("d", [4, 5, 8, 31, 32, 33, 64, 100])
def test_lloyd_step(d):
    """Clusters of 1 to several hundred members around well-separated centres."""
    rng = np.random.default_rng(d)
    k = 100
    centres = rng.normal(size=(k, d)) * 50
    sizes = np.concatenate([[1, 2, 7, 8, 9, 31, 32, 33, 64, 65, 300], rng.integers(1, 40, k - 11)])
    x = np.concatenate([centres[i] + 0.01 * rng.normal(size=(n, d)) for i, n in enumerate(sizes)]).astype(np.float32)
    x = np.ascontiguousarray(x[rng.permutation(len(x))])
    ivf = qb.IVFIndex(d, k, 8)
    ivf.train(x, max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)
    first = ivf.centroids()
    ivf = qb.IVFIndex(d, k, 8)
    ivf.train(x, max_iters=2, seed=1, clustering=qb.Clustering.Lloyd)
    second = ivf.centroids()
    d2 = ((x[:, None, :].astype(np.float64) - first[None]) ** 2).sum(2)
    if len(np.unique(d2.argmin(1))) < k:
        pytest.skip("a cluster without points (its refill has tests of its own)")
    assert lloyd_step(x, first, False).tobytes() == second.tobytes()
