"""The block-wide ranks behind the merge and the re-rank at the sizes where they
can go wrong: chunk counts and k' around the thread counts, empty entries, and
keys crowded into one interval (equal distances)."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


def merged(keys, slots, kp):
    import torch
    nq, nparts, _ = keys.shape
    k = torch.from_numpy(keys.view(np.int64)).cuda()
    s = torch.from_numpy(slots.view(np.int32)).cuda()
    ok = torch.empty(nq, kp, dtype=torch.int64, device="cuda")
    os_ = torch.empty(nq, kp, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    qb.merge_candidates_device(k.data_ptr(), s.data_ptr(), nq, nparts, kp, ok.data_ptr(), os_.data_ptr())
    return ok.cpu().numpy().view(np.uint64), os_.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("kp", [1, 2, 31, 100, 257, 1024, 3072])
@pytest.mark.parametrize("nparts", [1, 3, 32])
@pytest.mark.parametrize("kind", ["spread", "narrow", "one", "outlier", "empty"])
def test_merge(kp, nparts, kind):
    rng = np.random.default_rng(kp * 37 + nparts)
    for nq in (1, 5, 400):
        if nq == 400 and kp * nparts > 4000:
            continue
        n = nparts * kp
        high = {"spread": rng.integers(0, 2**32 - 1, (nq, n)), "narrow": rng.integers(2**31, 2**31 + 50, (nq, n)),
                "one": np.full((nq, n), 7), "outlier": np.where(rng.random((nq, n)) < 1.0 / n, 2**32 - 2, 1000) +
                rng.integers(0, 2, (nq, n)) * 0, "empty": rng.integers(0, 2**32 - 1, (nq, n))}[kind]
        low = np.stack([rng.permutation(n) for _ in range(nq)])
        keys = (high.astype(np.uint64) << np.uint64(32)) | low.astype(np.uint64)
        if kind == "empty":
            keys[rng.random((nq, n)) < 0.7] = np.uint64(2**64 - 1)
        slots = (low.astype(np.uint32) * np.uint32(3)) + np.uint32(1)
        want = np.sort(keys, axis=1)[:, :kp]
        got_k, got_s = merged(np.ascontiguousarray(keys.reshape(nq, nparts, kp)),
                              np.ascontiguousarray(slots.reshape(nq, nparts, kp)), kp)
        np.testing.assert_array_equal(got_k, want)
        live = want != np.uint64(2**64 - 1)
        want_s = ((want & np.uint64(0xFFFFFFFF)) * np.uint64(3) + np.uint64(1)).astype(np.uint32)
        np.testing.assert_array_equal(got_s[live], want_s[live])
        assert (got_s[~live] == 0xFFFFFFFF).all()


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("k,k_factor", [(1, 1), (7, 3), (10, 51), (10, 52), (100, 30)])
def test_refine_is_the_exact_order_of_its_candidates(metric, k, k_factor):
    """Every row a candidate (all lists probed, k' = live rows): the re-rank is the exact search."""
    n, d = k * k_factor, 24
    rng = np.random.default_rng(n)
    x = rng.normal(size=(max(n, 200), d)).astype(np.float32)[: max(n, 200)]
    x[: len(x) // 3] = x[0]   # ties, by slot
    ivf = qb.IVFIndex(d, 100, 100, metric=qb.Metric(metric))
    ivf.enable_pq(12, fast_scan=True)
    ivf.train(x if len(x) >= 100 else np.repeat(x, 3, axis=0), max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)
    idx = qb.RefineIndex(ivf, max(k_factor, -(-len(x) // k)))
    idx.add(x)
    flat = qb.FlatIndex(d, metric=qb.Metric(metric))
    flat.add(x)
    q = rng.normal(size=(33, d)).astype(np.float32)
    q[0] = 0.0   # scores of -0 or one value for all
    got, want = idx.batch_query(q, k), flat.batch_query(q, k)
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1].tobytes() == want[1].tobytes()
