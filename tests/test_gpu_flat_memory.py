"""Flat search on a card that is nearly full: without room for the rows' copy for the
tensor cores it goes through the exact tiles, with the same answers."""
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]

# 1,000,000 x 256 float32: 1,024 MB of rows, a copy of 516 MB; the exact tiles take 256 MB
CHILD = """
import numpy as np
import torch
import qann_b200 as qb

n, d, nq = 1_000_000, 256, 64
rng = np.random.default_rng(0)
x = rng.normal(size=(n, d)).astype(np.float32)
q = rng.normal(size=(nq, d)).astype(np.float32)

def answers():
    idx = qb.FlatIndex(d)
    idx.add(x)
    return idx.batch_query(q, 10), qb.tensor_filter_counts()["queries"]

small = qb.FlatIndex(4)
small.add(np.zeros((1, 4), np.float32))
small.batch_query(np.zeros((1, 4), np.float32), 1)   # (the context is up)
before = qb.tensor_filter_counts()["queries"]
# (added first: an add takes the rows to the card and gives the memory back to the library's pool)
idx = qb.FlatIndex(d)
idx.add(x)
free, _ = torch.cuda.mem_get_info()
hold = [torch.empty(free - (420 << 20), dtype=torch.uint8, device="cuda")]
got = idx.batch_query(q, 10)
assert qb.tensor_filter_counts()["queries"] == before, "made a copy after all"
hold.clear()
torch.cuda.empty_cache()
want, after = answers()
assert after == before + nq
assert (got[0] == want[0]).all() and got[1].tobytes() == want[1].tobytes()
print("the same")
"""


def test_nearly_full_card():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("the same"), r.stdout + r.stderr
