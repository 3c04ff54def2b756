"""Launches whose dynamic shared memory lies just below 48 KB and with the kernel's
static arrays above it, in a process that has asked for no more yet."""
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]

CHILD = """
import sys
import numpy as np
import qann_b200 as qb

n, k = int(sys.argv[1]), int(sys.argv[2])
x = np.random.default_rng(n).normal(size=(n, 4)).astype(np.float32)
idx = qb.FlatIndex(4)
idx.add(x)
qb.set_tensor_filter(0)   # the exact tiles and the row select
ids, d = idx.batch_query(x[:5], k)
assert (ids[:, 0] == np.arange(5)).all() and (np.diff(d, axis=1) >= 0).all()
print("fits")
"""


@pytest.mark.parametrize("n,k", [(12_216, 10), (12_100, 10), (11_900, 10), (8191, 700), (8100, 1000)])
def test_row_select(n, k):
    r = subprocess.run([sys.executable, "-c", CHILD, str(n), str(k)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("fits"), r.stdout + r.stderr
