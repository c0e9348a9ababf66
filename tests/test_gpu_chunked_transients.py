"""2-D bifurcation sweeps in chunks of the scratch budget whose transients run in
slices: the points of every chunk give what they give in one chunk, and the
chunks share the scratch of one."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
SWEEPS = {"lorenz": ([10.0, 28.0, 8 / 3], [0.1, 0.1, 0.1], [1, 0], [20.0, 200.0, 5.0, 15.0]),
          "chameleon": ([0.5, 3.0, 0.0, 2.0, 1.0, 18.0, 1.0], [3.0, 3.0, 0.0], [3, 5], [0.0, 5.0, 0.0, 20.0])}


# chunks of some 1.3 and 4.4 rows of 128 points per SM (152 of them) with 300 rows of intervals each
@pytest.mark.parametrize("system, n, budget", [("lorenz", 283, 122), ("chameleon", 420, 412)])
def test_chunks_with_sliced_transients(engine, monkeypatch, system, n, budget):
    values, start, mut, ranges = SWEEPS[system]
    kw = dict(tMax=6.005, nPts=n, h=0.01, initialConditions=start, ranges=ranges, indicesOfMutVars=mut,
              writableVar=0, maxValue=1e4, transientTime=200.0, values=values, eps=0.01, precision="fp32")
    engine.set_tuning(engine.TUNE_BIF2D_CAP, -1)
    try:
        whole = engine.bifurcation2d(system, **kw)
        monkeypatch.setenv("CHAOS_SCRATCH_BUDGET_MB", str(budget))
        before = engine.launch_count()
        chunked = engine.bifurcation2d(system, **kw)
    finally:
        engine.set_tuning(engine.TUNE_BIF2D_CAP, 0)
    assert engine.launch_count() - before > 2 * 4  # more than a sweep and a clustering launch for each of 3 or 4 chunks
    for k in whole:
        assert np.array_equal(np.asarray(whole[k]), np.asarray(chunked[k])), k
    assert (np.asarray(whole["counts"]) > 0).sum() > 100


GROWTH = """
import os, sys
os.environ["CHAOS_SCRATCH_BUDGET_MB"] = "19"
sys.path.insert(0, {root!r})
import torch
import chaoslibrary_gb300 as C

def run(n):
    out = dict(labels=torch.zeros(n * n, dtype=torch.int32, device="cuda"),
               counts=torch.zeros(n * n, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    before = C.launch_count()
    C.bifurcation2d("lorenz", 1.205, n, 0.01, [0.1, 0.1, 0.1], [20.0, 200.0, 5.0, 15.0], [1, 0], 0, 1e4, 40.0,
                    [10.0, 28.0, 8 / 3], 1, 0.01, precision="fp32", out=out)
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0], C.launch_count() - before

run(16)
grown, launches = run(4000)
print("grown", grown, launches)
"""


def test_chunks_share_their_scratch():
    """16,000,000 points in some 780 chunks of 19 MB: the states of all of them would be 256 MB."""
    r = subprocess.run([sys.executable, "-c", GROWTH.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    grown, launches = (int(v) for v in r.stdout.split()[-2:])
    assert launches > 3 * 700  # the transients ran in slices
    assert grown < 96 << 20
