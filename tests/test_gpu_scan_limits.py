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
