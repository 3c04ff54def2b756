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


def both(fn):
    qb.set_tensor_filter(0)
    exact = fn()
    qb.set_tensor_filter(2)
    got, queries, redone = tensor_redone(fn)
    np.testing.assert_array_equal(exact[0], got[0])
    assert exact[1].tobytes() == got[1].tobytes()
    return queries, redone


@pytest.mark.parametrize("d", [1, 7, 63, 65, 96, 128, 129, 300, 768, 2048])
@pytest.mark.parametrize("metric", [0, 1, 2])
def test_flat_tile_edges(d, metric):
    """Row counts around the seed and the tiles, queries around a half tile, k from 1 to the engine's largest."""
    for n, nq, k in ((100, 3, 100), (2047, 129, 10), (2049, 256, 1), (9000, 257, 40), (9001, 5, 1024)):
        idx = qb.FlatIndex(d, metric=qb.Metric(metric))
        idx.add(rows_of("normal", d + n, n, d))
        q = rows_of("normal", d + n + 1, nq, d)
        queries, redone = both(lambda: idx.batch_query(q, k))
        assert queries == nq
        if d >= 96:
            assert redone == 0


@pytest.mark.parametrize("kind", ["mixture", "duplicates", "positive", "scales", "tiny", "huge", "odd_rows"])
@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("warps", [8, 16])
def test_flat_data(kind, metric, warps):
    d, n = 100, 20_000
    idx = qb.FlatIndex(d, metric=qb.Metric(metric))
    idx.add(rows_of(kind, 8, n, d))
    q = rows_of(kind, 9, 200, d)
    qb.set_filter_options(epilogue_warps=warps)
    for k in (1, 10, 100):
        both(lambda: idx.batch_query(q, k))
    idx.remove(np.arange(0, n, 5))
    both(lambda: idx.batch_query(q, 10))
    allowed = np.arange(0, n, 301)
    both(lambda: idx.batch_query(q, 100, allowed=allowed))   # fewer allowed than wanted


def test_flat_sorted_rows():
    """Rows stored nearest last: every chunk holds more near rows than the one before it."""
    d, n = 32, 60_000
    rng = np.random.default_rng(3)
    x = (rng.normal(size=(n, d)) * np.linspace(4.0, 0.1, n)[:, None]).astype(np.float32)
    idx = qb.FlatIndex(d)
    idx.add(x)
    q = (0.1 * rng.normal(size=(70, d))).astype(np.float32)
    both(lambda: idx.batch_query(q, 50))


def test_flat_non_finite():
    """Infinite and NaN components rank as the exact path ranks them."""
    d, n = 48, 9000
    x = rows_of("normal", 1, n, d)
    x[5, 3] = np.inf
    x[77, 0] = -np.inf
    x[100, 1] = np.nan
    idx = qb.FlatIndex(d)
    idx.add(x)
    q = rows_of("normal", 2, 66, d)
    for k in (1, 20):
        both(lambda: idx.batch_query(q, k))
    q[3, 2] = np.inf
    q[9, 7] = 1e30
    both(lambda: idx.batch_query(q, 20))


@pytest.mark.parametrize("d,m", [(129, None), (256, 64), (768, 64)])
@pytest.mark.parametrize("metric", [0, 2])
def test_coarse_wide(d, m, metric):
    """The coarse step of dimensions past 128 on the tensor cores."""
    if m is None:
        d, m = 130, 26
    x = rows_of("mixture", d, 20_000, d)
    ivf = qb.IVFIndex(d, 400, 8, metric=qb.Metric(metric))
    ivf.enable_pq(m, fast_scan=True)
    ivf.train(x, max_iters=2, seed=5, clustering=qb.Clustering.Lloyd)
    ivf.add(x)
    q = rows_of("mixture", d + 1, 300, d)
    for nprobe in (1, 40):
        ivf.nprobe = nprobe
        qb.set_tensor_filter(0)
        exact = ivf.batch_query(q, 10)
        qb.set_tensor_filter(2)
        before = qb.tensor_filter_counts()["coarse_queries"]
        got = ivf.batch_query(q, 10)
        assert qb.tensor_filter_counts()["coarse_queries"] - before == 300
        np.testing.assert_array_equal(exact[0], got[0])
        assert exact[1].tobytes() == got[1].tobytes()


def test_flat_kept_copy_follows_the_rows():
    """The f16 copy kept with a FlatIndex is made again after rows are added or removed."""
    d = 64
    x = rows_of("normal", 4, 50_000, d)
    q = rows_of("normal", 5, 9, d)
    idx = qb.FlatIndex(d)
    idx.add(x[:30_000])
    both(lambda: idx.batch_query(q, 10))
    idx.add(x[30_000:] * np.float32(0.01))
    both(lambda: idx.batch_query(q, 10))
    idx.remove(np.arange(30_000, 50_000, 2))
    both(lambda: idx.batch_query(q, 10))
    refine = qb.RefineIndex(qb.FlatIndex(d), 4)
    refine.add(x)
    both(lambda: refine.batch_query(q, 10))


def test_flat_concurrent_first_searches():
    """Threads that search a fresh FlatIndex at the same time get the same answers (one of them makes the copy)."""
    import threading
    d = 48
    x = rows_of("mixture", 6, 60_000, d)
    q = rows_of("mixture", 7, 40, d)
    qb.set_tensor_filter(0)
    ref = qb.FlatIndex(d)
    ref.add(x)
    want = ref.batch_query(q, 10)
    qb.set_tensor_filter(2)
    idx = qb.FlatIndex(d)
    idx.add(x)
    got = [None] * 4
    def work(i):
        got[i] = idx.batch_query(q, 10)
    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for g in got:
        np.testing.assert_array_equal(g[0], want[0])
        assert g[1].tobytes() == want[1].tobytes()


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("nq,k", [(1, 1), (149, 10), (400, 10), (1200, 9), (1200, 100)])
def test_one_copy_results(metric, nq, k):
    """Small results come back in one copy, larger ones apart; from device
    buffers (whatever their alignment) the same bits, coarse step either way."""
    import torch
    d = 40
    x = rows_of("mixture", 12, 20_000, d)
    ivf = qb.IVFIndex(d, 300, 20, metric=qb.Metric(metric))
    ivf.enable_pq(20, fast_scan=True)
    ivf.train(x, max_iters=2, seed=5, clustering=qb.Clustering.Lloyd)
    idx = qb.RefineIndex(ivf, 4)
    idx.add(x)
    q = rows_of("mixture", 13, nq, d)
    q[0] *= np.float32(1e-12)   # a norm its coarse bounds do not hold for
    qb.set_tensor_filter(0)
    want = idx.batch_query(q, k)
    for mode in (1, 2):
        qb.set_tensor_filter(mode)
        got = idx.batch_query(q, k)
        np.testing.assert_array_equal(got[0], want[0])
        assert got[1].tobytes() == want[1].tobytes()
        pad = torch.zeros(nq * d + 1, device="cuda")
        pad[1:] = torch.from_numpy(q).cuda().ravel()   # rows 4 bytes off
        ids = torch.empty(nq, k, dtype=torch.int64, device="cuda")
        dist = torch.empty(nq, k, device="cuda")
        idx.search_device(pad.data_ptr() + 4, nq, k, ids.data_ptr(), dist.data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
        np.testing.assert_array_equal(ids.cpu().numpy(), want[0])
        assert dist.cpu().numpy().tobytes() == want[1].tobytes()
