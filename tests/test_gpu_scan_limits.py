"""The scan at the end of what its shared memory holds: tables per list from the
query itself (precomputed_tables off) take `dim` floats of it."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


def wide_index(d, m, n=150, nlist=100):
    rng = np.random.default_rng(d)
    x = rng.normal(size=(n, d)).astype(np.float32)
    ivf = qb.IVFIndex(d, nlist, nlist)
    ivf.enable_pq(m, fast_scan=True)
    ivf.precomputed_tables = False
    ivf.train(x, max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)
    ivf.add(x)
    return ivf, rng.normal(size=(2, d)).astype(np.float32)


@pytest.mark.parametrize("variant", [-1, 0, 1, 2])
def test_no_shape_fits(variant):
    """More dims than any block can hold: refused, under every choice of shapes."""
    ivf, q = wide_index(61_440, 1024)
    qb.set_scan_options(variant=variant)
    try:
        with pytest.raises(RuntimeError, match="shared memory"):
            ivf.batch_query(q, 10)
    finally:
        qb.set_scan_options(variant=-1)


@pytest.mark.parametrize("k", [1, 10, 100])
def test_last_that_fits(k, tmp_path):
    """The most dims one warp's block holds beside its buffer of k' + 256 keys
    (226 KB with units of 8 probes, in steps of 16 dims), against the oracle's
    scan of the saved lists."""
    from oracle import qann_file

    d, m = {1: 56_816, 10: 56_816, 100: 56_512}[k], 16
    ivf, q = wide_index(d, m)
    ivf.nprobe = 8
    ids, dist = ivf.batch_query(q, k)
    ivf.save(tmp_path / "wide.qann")
    info = qann_file.read(tmp_path / "wide.qann")["ivf"]
    arr = qann_file.arrays(info)
    for i in range(len(q)):
        probes, pterm = qann_file.coarse(info, q[i], info["nprobe"])
        want_d, want_s = arr.query(q[i], probes, pterm, k)
        order = np.lexsort((want_s, want_d))
        n = len(order)   # (8 lists hold fewer than 100 vectors)
        np.testing.assert_array_equal(ids[i, :n], want_s[order].astype(np.int64))
        assert dist[i, :n].tobytes() == want_d[order].tobytes()
        assert (ids[i, n:] == -1).all()
