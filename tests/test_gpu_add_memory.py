"""Adding wide rows on a card that is nearly full: they are prepared for the tensor
cores a block of at most 256 MB at a time."""
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]

# 200,000 x 2,048 float32: 1,638 MB of rows, 820 MB if all are prepared at once;
# candidate lists 268 MB
CHILD = """
import sys
import numpy as np
import torch
import qann_b200 as qb

n, d, nlist = 200_000, 2048, 100
rng = np.random.default_rng(0)
x = np.tile(rng.normal(size=(n // 20, d)).astype(np.float32), (20, 1)) * np.linspace(1, 2, n, dtype=np.float32)[:, None]

def index():
    ivf = qb.IVFIndex(d, nlist, 8)
    ivf.enable_pq(2, fast_scan=True)
    ivf.train(x[:: n // 2000], max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)
    return ivf

def saved(ivf):
    ivf.add(x)
    ivf.save(sys.argv[1])
    return open(sys.argv[1], "rb").read()

ivf = index()
free, _ = torch.cuda.mem_get_info()
hold = [torch.empty(free - (2450 << 20), dtype=torch.uint8, device="cuda")]
full = saved(ivf)
hold.clear()
torch.cuda.empty_cache()
assert saved(index()) == full
print("the same")
"""


def test_nearly_full_card(tmp_path):
    r = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "a.qann")], cwd=ROOT, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and r.stdout.strip().endswith("the same"), r.stdout + r.stderr
