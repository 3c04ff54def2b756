"""Rows made unit length (32 a block, 32 columns at a time), at the widths and
counts around those numbers: added rows and queries against a float64 sum in
index order, and zero rows."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu

WIDTHS = [1, 2, 31, 32, 33, 64, 65, 100, 129]


def unit(x):
    """x / |x| as the library forms it: squares summed one after the other in
    float64 (a float's square is exact there), one float scale per row."""
    s = np.zeros(len(x), np.float64)
    for c in range(x.shape[1]):
        v = x[:, c].astype(np.float64)
        s = s + v * v
    return x * (1.0 / np.sqrt(s)).astype(np.float32)[:, None]


def rows_of(n, d, seed):
    rng = np.random.default_rng(seed)
    x = (rng.normal(size=(n, d)) * np.exp(rng.normal(0, 3, (n, 1)))).astype(np.float32)
    x[0] = 0.0
    x[0, d - 1] = 3.0    # all of the norm in the last column
    x[n // 2, 1:] = 0.0  # or the first
    x[n // 2, 0] = -0.5
    return x


@pytest.mark.parametrize("d", WIDTHS)
@pytest.mark.parametrize("n", [128, 159, 161, 1000])
def test_added_rows(d, n, tmp_path):
    x = rows_of(n, d, 100 * d + n)
    idx = qb.FlatIndex(d, metric=qb.Metric.Cosine)
    idx.add(x)
    idx.save(tmp_path / "unit.qann")
    assert unit(x).tobytes() in (tmp_path / "unit.qann").read_bytes()   # the file holds the rows as they are


@pytest.mark.parametrize("d", WIDTHS)
@pytest.mark.parametrize("nq", [1, 31, 32, 33, 97])
def test_queries(d, nq):
    """A cosine score is half the squared distance of the unit rows, to the bit."""
    x, q = rows_of(200, d, d), rows_of(max(nq, 2), d, 7 * d)[:nq]
    a, b = qb.FlatIndex(d, metric=qb.Metric.Cosine), qb.FlatIndex(d)
    a.add(x)
    b.add(unit(x))
    got, want = a.batch_query(q, 5), b.batch_query(unit(q), 5)
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1].tobytes() == (want[1] * np.float32(0.5)).tobytes()


@pytest.mark.parametrize("at", [0, 31, 32, 99])
def test_zero_rows_are_refused(at):
    x = rows_of(100, 33, 5)
    idx = qb.FlatIndex(33, metric=qb.Metric.Cosine)
    idx.add(x)
    x[at] = 0.0
    with pytest.raises(ValueError, match="non-zero"):
        idx.add(x)
    with pytest.raises(ValueError, match="non-zero"):
        idx.batch_query(x, 1)
    assert len(idx) == 100
