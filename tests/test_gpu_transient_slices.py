"""FP32 sweeps whose transient runs in slices, with the points' states in
scratch in between, give what the same sweep gives in one launch (a captured
stream, or a scratch budget below the states): just over one, two and four rows
of 128 points per SM with a ragged end, a transient that is no multiple of the
slices, orbits that diverge in it or come to rest, each recorded component."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SWEEPS = {"lorenz": ([10.0, 28.0, 8 / 3], [0.1, 0.1, 0.1], [1], [0.5, 200.0]),
          "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 1.0], [2], [2.0, 10.0]),
          "chen": ([35.0, 3.0, 28.0], [-10.0, 0.0, 37.0], [2], [20.0, 30.0]),
          "chameleon": ([0.5, 3.0, 0.0, 2.0, 1.0, 18.0, 1.0], [3.0, 3.0, 0.0], [3], [0.0, 5.0])}


@pytest.mark.parametrize("system", sorted(SWEEPS))
@pytest.mark.parametrize("rows, wv, max_value, transient", [(1, 0, 1e4, 250.03), (2, 1, 12.0, 100.0), (4, 2, 1e4, 81.7),
                                                             (4, 0, 1e4, 400.0)])
def test_sliced_transient_of_a_bifurcation(engine, system, rows, wv, max_value, transient):
    import torch

    values, ic, mut, rg = SWEEPS[system]
    n = rows * 128 * torch.cuda.get_device_properties(0).multi_processor_count + 131
    z = lambda shape, t: torch.zeros(shape, dtype=t, device="cuda")  # noqa: E731
    out = dict(counts=z(n, torch.int32), flags=z(n, torch.int32), first=z(n, torch.float64),
               peaks=z((n, 24), torch.float64), intervals=z((n, 24), torch.float64))

    def run():
        before = engine.launch_count()
        engine.bifurcation1d(system, 10.0, n, 0.01, ic, rg, mut, wv, max_value, transient, values, peakCapacity=24,
                             precision="fp32", out=out)
        return engine.launch_count() - before

    launches = run()
    assert launches > 1 or system == "chameleon" or transient < 200.0  # where slices certainly pay
    torch.cuda.synchronize()
    sliced = {k: v.cpu().numpy() for k, v in out.items()}
    for v in out.values():
        v.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert run() == 1
    graph.replay()
    torch.cuda.synchronize()
    for k, v in out.items():
        assert np.array_equal(sliced[k], v.cpu().numpy(), equal_nan=True), k


@pytest.mark.parametrize("system", ["lorenz", "rossler"])
@pytest.mark.parametrize("pre", [1, 2])
def test_sliced_transient_of_basins(engine, monkeypatch, system, pre):
    values, ic, _, _ = SWEEPS[system]
    n = 283  # 80,089 points: 4.1 rows on 152 SMs, more states than a megabyte holds
    kw = dict(tMax=20.0, nPts=n, h=0.01, initialConditions=ic, ranges=[-30.0, 30.0, -30.0, 30.0],
              indicesOfMutVars=[0, 1], writableVar=0, maxValue=1e8, transientTime=400.0, values=values,
              preScaller=pre, eps=0.05, precision="fp32")
    before = engine.launch_count()
    a = engine.basins(system, **kw)
    sliced = engine.launch_count() - before
    monkeypatch.setenv("CHAOS_SCRATCH_BUDGET_MB", "1")
    before = engine.launch_count()
    b = engine.basins(system, **kw)
    assert sliced > engine.launch_count() - before
    for k in a:
        assert np.array_equal(np.asarray(a[k]), np.asarray(b[k]), equal_nan=True), k


def test_sliced_transient_of_a_2d_sweep(engine, monkeypatch):
    values, ic, _, _ = SWEEPS["chameleon"]
    kw = dict(tMax=40.0, nPts=283, h=0.01, initialConditions=ic, ranges=[0.0, 5.0, 0.0, 20.0], indicesOfMutVars=[3, 5],
              writableVar=0, maxValue=1e4, transientTime=500.0, values=values, eps=0.001, precision="fp32")
    a = engine.bifurcation2d("chameleon", **kw)
    monkeypatch.setenv("CHAOS_SCRATCH_BUDGET_MB", "1")
    b = engine.bifurcation2d("chameleon", **kw)
    for k in a:
        assert np.array_equal(np.asarray(a[k]), np.asarray(b[k])), k
