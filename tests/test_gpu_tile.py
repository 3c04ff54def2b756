"""The tensor-core tile engine against the exact paths, at the edges of its
tiles (256 queries x 128 rows, K blocks of 64) and on the data its bounds have
to hold for: ties, unequal scales, zero, huge, tiny and non-finite rows."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def default_mode():
    yield
    qb.set_tensor_filter(1)
    qb.set_filter_options(autotune=True, epilogue_warps=0)


def rows_of(kind, seed, n, d):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, d)).astype(np.float32)
    if kind == "mixture":
        c = rng.normal(size=(60, d)).astype(np.float32)
        x = c[rng.integers(0, 60, n)] + np.float32(0.2) * x
    elif kind == "duplicates":
        x = x[rng.integers(0, max(1, n // 3), n)]
    elif kind == "positive":
        x = np.abs(x) + np.float32(3.0)
    elif kind == "scales":   # norms from 1e-6 to 1e6
        x *= (10.0 ** rng.uniform(-6, 6, (n, 1))).astype(np.float32)
    elif kind == "tiny":
        x *= np.float32(1e-9)
    elif kind == "huge":
        x *= np.float32(1e12)
    elif kind == "odd_rows":   # zero rows, rows whose squares under- and overflow
        x[rng.integers(0, n, max(1, n // 50))] = 0.0
        x[rng.integers(0, n, max(1, n // 60))] *= np.float32(1e-22)
        x[rng.integers(0, n, max(1, n // 60))] *= np.float32(1e17)
    return np.ascontiguousarray(x)


def lloyd(x, nlist):
    ivf = qb.IVFIndex(x.shape[1], nlist, 8)
    ivf.train(x, max_iters=2, seed=3, clustering=qb.Clustering.Lloyd)
    return ivf.centroids().tobytes()


def tensor_redone(fn):
    before = qb.tensor_filter_counts()
    out = fn()
    after = qb.tensor_filter_counts()
    return out, after["queries"] - before["queries"], after["redone"] - before["redone"]


@pytest.mark.parametrize("d", [1, 7, 16, 63, 64, 65, 100, 128, 129, 200, 515, 2048])
@pytest.mark.parametrize("n,nlist", [(1023, 127), (1025, 129), (700, 385), (256, 128)])
def test_nearest_tile_edges(d, n, nlist):
    """Lloyd's centroids depend on every label: the same bytes either way."""
    x = rows_of("normal", d, n, d)
    qb.set_tensor_filter(0)
    exact = lloyd(x, nlist)
    qb.set_tensor_filter(2)
    got, queries, redone = tensor_redone(lambda: lloyd(x, nlist))
    assert got == exact
    assert queries >= 3 * n
    if d >= 16:   # (low dimensions are crowded: rows within the bound of one another overflow)
        assert redone <= 0.02 * queries


@pytest.mark.parametrize("kind", ["mixture", "duplicates", "positive", "scales", "tiny", "huge", "odd_rows"])
@pytest.mark.parametrize("warps", [8, 16])
@pytest.mark.parametrize("d", [24, 100, 300])
def test_nearest_data(kind, warps, d):
    x = rows_of(kind, 5, 6000, d)
    qb.set_tensor_filter(0)
    exact = lloyd(x, 500)
    qb.set_tensor_filter(2)
    qb.set_filter_options(epilogue_warps=warps)
    assert lloyd(x, 500) == exact
