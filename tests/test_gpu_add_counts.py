"""Adds on either side of the size up to which vectors go to their lists one by one:
the saved index is the same however the rows are divided into adds."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("custom", [False, True])
def test_same_lists_however_added(metric, custom, tmp_path):
    rng = np.random.default_rng(metric)
    n, d = 12_000, 24
    x = rng.normal(size=(n, d)).astype(np.float32)
    ids = rng.permutation(3 * n)[:n].astype(np.int64)

    def saved(sizes):
        ivf = qb.IVFIndex(d, 128, 8, metric=qb.Metric(metric), custom_ids=custom)
        ivf.enable_pq(12, fast_scan=True)
        ivf.train(x[:3000], max_iters=2, seed=1, clustering=qb.Clustering.Lloyd)
        at = 0
        for s in sizes:
            ivf.add(x[at:at + s], *([ids[at:at + s]] if custom else []))
            at += s
        assert at == n
        ivf.save(tmp_path / "a.qann")
        return (tmp_path / "a.qann").read_bytes()

    whole = saved([n])
    assert saved([4096, 4097, 1, 63, n - 8257]) == whole
    assert saved([1, 2, 4095, n - 4098]) == whole
    assert saved([1000] * 12) == whole
