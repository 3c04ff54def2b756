"""Flat search over rows stored in an order: what is near comes all at once, more of
it than a query's candidate list takes. The answers are the exact path's, and the
queries stay on the tensor cores (sweeps with falling thresholds) but for ties that
no list holds."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def default_mode():
    yield
    qb.set_tensor_filter(1)


def rows_of(kind, n, d, nq):
    rng = np.random.default_rng(n + d)
    if kind == "near_last":    # each row nearer than the ones before it
        x = rng.normal(size=(n, d)).astype(np.float32) * np.linspace(3.0, 0.3, n, dtype=np.float32)[:, None]
        return x, (0.3 * rng.normal(size=(nq, d))).astype(np.float32)
    c = rng.normal(size=(25, d)).astype(np.float32)
    lab = np.sort(rng.integers(0, 25, n))
    spread = {"clusters": 0.3, "tight": 1e-3, "ties": 0.0}[kind]
    x = c[lab] + np.float32(spread) * rng.normal(size=(n, d)).astype(np.float32)
    q = c[rng.integers(0, 25, nq)] + np.float32(0.2) * rng.normal(size=(nq, d)).astype(np.float32)
    return x, q


def both(fn):
    """The exact path's answer and the tensor cores', which must be the same; the
    queries that went on to the exact path after all."""
    qb.set_tensor_filter(0)
    want = fn()
    qb.set_tensor_filter(2)
    before = qb.tensor_filter_counts()
    got = fn()
    after = qb.tensor_filter_counts()
    qb.set_tensor_filter(1)
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1].tobytes() == want[1].tobytes()
    return after["redone"] - before["redone"]


@pytest.mark.parametrize("kind", ["near_last", "clusters"])
@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("nq,k", [(1, 10), (1, 1), (64, 100), (65, 10), (300, 257), (40, 600), (20, 1024)])
def test_settled_without_the_exact_path(kind, metric, nq, k):
    x, q = rows_of(kind, 200_000, 48, nq)
    idx = qb.FlatIndex(48, metric=qb.Metric(metric))
    idx.add(x)
    assert both(lambda: idx.batch_query(q, k)) == 0


@pytest.mark.parametrize("n", [190_000, 250_000])
@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("nq,k", [(1, 10), (64, 100), (20, 1024)])
def test_ties(metric, nq, k, n):
    """7,600 equal rows fit a sweep's list of 8,192; 10,000 do not, and go on."""
    x, q = rows_of("ties", n, 32, nq)
    idx = qb.FlatIndex(32, metric=qb.Metric(metric))
    idx.add(x)
    redone = both(lambda: idx.batch_query(q, k))
    assert redone == 0 if n == 190_000 else redone <= nq
    x, q = rows_of("tight", n, 32, nq)
    idx = qb.FlatIndex(32, metric=qb.Metric(metric))
    idx.add(x)
    both(lambda: idx.batch_query(q, k))


def test_filters_deletions_and_odd_queries():
    d, n = 40, 150_000
    x, q = rows_of("clusters", n, d, 90)
    x[7, 3] = np.inf
    x[n - 9, 0] = np.nan
    x[n // 2] = 0.0
    x[n // 3] *= np.float32(1e25)
    idx = qb.FlatIndex(d)
    idx.add(x)
    q[4] = 0.0
    q[5, 2] = np.nan
    q[6] *= np.float32(1e30)
    q[7] *= np.float32(1e-30)
    rng = np.random.default_rng(0)
    both(lambda: idx.batch_query(q, 20))
    allowed = np.sort(rng.choice(n, n // 2, replace=False))
    both(lambda: idx.batch_query(q, 20, allowed=allowed))
    both(lambda: idx.batch_query(q[:1], 100, allowed=allowed[-50:]))
    idx.remove(allowed)
    both(lambda: idx.batch_query(q, 20))


def test_rows_past_one_launch():
    """More rows than a launch of the tile kernel takes (2^22)."""
    d, n = 8, (1 << 22) + 12_345
    rng = np.random.default_rng(1)
    x = rng.normal(size=(n, d)).astype(np.float32) * np.linspace(3.0, 1.0, n, dtype=np.float32)[:, None]
    idx = qb.FlatIndex(d)
    idx.add(x)
    q = rng.normal(size=(3, d)).astype(np.float32)
    both(lambda: idx.batch_query(q, 30))


@pytest.mark.parametrize("k,seed", [(10, 2048), (200, 3200), (700, 8192)])
@pytest.mark.parametrize("d", [20, 136])
def test_around_the_sample(k, seed, d):
    """Row counts around one, two and three times the sample, whose step changes there."""
    rng = np.random.default_rng(seed + d)
    for n in [m * seed + e for m in (1, 2, 3) for e in (-1, 0, 1, 129)]:
        x = rng.normal(size=(n, d)).astype(np.float32)
        x = x[np.argsort(x[:, 0])]
        q = rng.normal(size=(67, d)).astype(np.float32)
        for metric in (qb.Metric.L2, qb.Metric.InnerProduct):
            idx = qb.FlatIndex(d, metric=metric)
            idx.add(x)
            idx.remove(np.arange(0, n, 7))
            for nq in (1, 67):
                both(lambda: idx.batch_query(q[:nq], k))
