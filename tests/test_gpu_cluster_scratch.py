"""Scratch of a large clustering: what is kept per sorted point is sized by the
points that were sorted, which in a set that settled on a few attractors are
few."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
GROWTH = """
import sys
sys.path.insert(0, {root!r})
import torch
import chaoslibrary_gb300 as C

def run(n):
    g = torch.Generator(device="cuda").manual_seed(0)
    X = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64) * 0.002
    X += (torch.arange(n, device="cuda") % 4)[:, None] * 0.25
    X[::100000] = torch.rand(len(X[::100000]), 3, generator=g, device="cuda", dtype=torch.float64)
    labels = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    C.dbscan(X, 0.05, 8, out=labels)
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0], [int(labels[k]) for k in range(1, 5)]

run(1000)
grown, labels = run({n})
print(grown, *labels)
"""


def test_scratch_per_point():
    n = 1 << 24
    r = subprocess.run([sys.executable, "-c", GROWTH.format(root=str(ROOT), n=n)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    grown, *labels = (int(v) for v in r.stdout.split())
    assert len(set(labels)) == 4 and min(labels) >= 0
    # a slot, an order, a cell, three coordinates and a mark per point are 37 B
    assert grown < 45 * n, grown / n


@pytest.mark.parametrize("d", [2, 3])
def test_large_set_against_a_small_one(engine, d):
    """Above the size at which the count of sorted points is waited for, a set
    made of copies of a small one far apart has the small one's labels in each."""
    import torch

    rng = np.random.default_rng(d)
    m, copies = 30000, 150  # 4,500,000 points
    X = np.concatenate([c + 0.01 * rng.standard_normal((m // 5, d)) for c in rng.uniform(0, 1, (4, d))] +
                       [rng.uniform(0, 1, (m - 4 * (m // 5), d))])
    X = np.round(X[rng.permutation(m)] * 2.0**30) / 2.0**30  # a shift by whole numbers is exact
    X = torch.tensor(X, device="cuda")
    for min_pts in (4, 40):
        small = engine.dbscan(X, 0.01, min_pts)
        shift = torch.zeros(copies, 1, d, dtype=torch.float64, device="cuda")
        shift[:, 0, 0] = 4.0 * torch.arange(copies, device="cuda")
        big = engine.dbscan((X[None] + shift).reshape(-1, d).contiguous(), 0.01, min_pts).reshape(copies, m)
        torch.cuda.synchronize()
        k = int(small.max()) + 1
        assert torch.equal(big[0], small)
        assert torch.equal(big >= 0, (small >= 0).expand(copies, m))
        rows = torch.arange(copies, dtype=torch.int32, device="cuda")[:, None] * k + small[None]
        assert torch.equal(torch.where(big >= 0, big, -1), torch.where(small[None] >= 0, rows, -1))
