"""LLE maps and spectra that run in slices of the horizon, with the points'
states in scratch in between, give the bits of the same call in one launch --
which is what a captured stream gets: just over one, two, four and eight rows
of 128 points per SM, with a ragged last block and an odd last point, without
a transient, with little else, with one step a block, and with a number of
blocks that is no multiple of the spectrum's groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYSTEMS = {"lorenz": ([10.0, 28.0, 8 / 3], [1.0, 1.0, 1.0], [1], [20.0, 200.0]),
           "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 1.0], [2], [2.0, 10.0]),
           "chen": ([35.0, 3.0, 28.0], [-10.0, 0.0, 37.0], [2], [20.0, 30.0])}


@pytest.mark.parametrize("system", sorted(SYSTEMS))
@pytest.mark.parametrize("kind, precision", [("lle", "fp32"), ("lle", "ff32"), ("spectrum", "fp32")])
@pytest.mark.parametrize("rows, tMax, NT, transient",
                         [(1, 60.0, 0.1, 5.0), (2, 47.3, 0.1, 0.0), (4, 31.0, 0.01, 2.5), (8, 40.0, 0.23, 40.0),
                          (1, 10.0, 2.0, 150.0), (4, 150.0, 0.01, 2.5), (8, 150.0, 0.23, 40.0)])
def test_slices_match_one_launch(engine, system, kind, precision, rows, tMax, NT, transient):
    import torch

    values, ic, mut, rg = SYSTEMS[system]
    n = rows * 128 * torch.cuda.get_device_properties(0).multi_processor_count + 131
    call = engine.lle_sweep if kind == "lle" else engine.lyapunov_spectrum
    out = torch.zeros(n * (1 if kind == "lle" else 3), dtype=torch.float64, device="cuda")

    def run():
        before = engine.launch_count()
        call(system, 1, tMax, NT, n, 0.01, 1e-8, ic, rg, mut, transient, values, precision=precision, out=out)
        return engine.launch_count() - before

    launches = run()
    assert launches > 1 or tMax < 45.0  # too short a horizon may run in one launch
    torch.cuda.synchronize()
    sliced = out.cpu().numpy()
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert run() == 1
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(sliced.view(np.int64), out.cpu().numpy().view(np.int64))
    assert np.isfinite(sliced).mean() > 0.5


def test_slices_of_a_map_match_single_points(engine):
    """A 2-D map in slices has the values of its single-point calls."""
    values, ic, mut, rg = SYSTEMS["lorenz"]
    n = 151  # just over one row on 152 SMs
    kw = dict(h=0.01, eps=1e-8, initialConditions=ic, transientTime=3.0, values=values, precision="fp32")
    big = engine.lle2d("lorenz", 80.0, 0.1, n, indicesOfMutVars=[1, 0], ranges=[20.0, 200.0, 5.0, 15.0], **kw)
    s0, s1 = 180.0 / (n - 1), 10.0 / (n - 1)
    for j, i in ((0, 0), (64, 7), (128, 150), (150, 150)):
        one = engine.lle2d("lorenz", 80.0, 0.1, 2, indicesOfMutVars=[1, 0],
                           ranges=[20.0 + i * s0, 300.0, 5.0 + j * s1, 20.0], **kw)
        assert np.asarray(one).reshape(-1)[0] == np.asarray(big).reshape(n, n)[j, i], (j, i)
