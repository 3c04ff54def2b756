"""Training on a card that is nearly full: the points' copy for the tensor cores is
kept only where there is room, and made a block of rows at a time otherwise."""
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]

# 20,000,000 x 2 float32: 160 MB of points, 480 MB as padded rows for the tensor
# cores; labels and order 160 MB, candidate lists 268 MB. 850 MB hold all but the copy.
CHILD = """
import numpy as np
import torch
import qann_b200 as qb

n, d, k = 20_000_000, 2, 100
rng = np.random.default_rng(0)
x = rng.normal(size=(n, d)).astype(np.float32)

def centroids():
    ivf = qb.IVFIndex(d, k, 8)
    ivf.train(x, max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)
    return ivf.centroids().tobytes()

qb.IVFIndex(d, k, 8).train(x[:1000], max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)   # (the context is up)
free, _ = torch.cuda.mem_get_info()
hold = [torch.empty(free - (850 << 20), dtype=torch.uint8, device="cuda")]
full = centroids()
hold.clear()
torch.cuda.empty_cache()
assert centroids() == full
print("the same")
"""


def test_nearly_full_card():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("the same"), r.stdout + r.stderr
