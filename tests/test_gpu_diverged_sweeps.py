"""Points that are beyond the bound when they begin to be recorded end at their
second sample: a map of such points costs its transient and little more,
however many samples were asked for and however many steps a sample takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision, mode, n", [("fp32", 2, 600), ("fp64", 0, 150)])
@pytest.mark.parametrize("system, values, start", [("lorenz", [10.0, 28.0, 8 / 3], [0.0, 0.0, 27.0]),
                                                   ("chen", [35.0, 3.0, 28.0], [0.0, 0.0, 20.0])])
def test_maps_that_diverged_in_the_transient(engine, precision, mode, n, system, values, start):
    import torch

    z = lambda t: torch.zeros(n * n, dtype=t, device="cuda")  # noqa: E731
    out = dict(flags=z(torch.int32), avg_peaks=z(torch.float64), avg_intervals=z(torch.float64), counts=z(torch.int32))

    def seconds(samples):
        """500 steps a sample; no transient, every start beyond the bound, where z stays."""
        best = 1e9
        for _ in range(5):
            t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            t[0].record()
            engine.basins_features(system, samples * 5.0 + 0.001, n, 0.01, start, [5.0, 20.0, 5.0, 20.0], [0, 1], 2,
                                   1e-3, 0.0, values, preScaller=500, precision=precision, out=out)
            t[1].record()
            torch.cuda.synchronize()
            best = min(best, t[0].elapsed_time(t[1]))
        assert (out["flags"].cpu().numpy() == 0).all()
        return best

    engine.set_tuning(engine.TUNE_SWEEP_PAIRS, mode)
    try:
        few = seconds(2)
        many = seconds(400)
    finally:
        engine.set_tuning(engine.TUNE_SWEEP_PAIRS, 1)
    # one sample each; a window would run 24 or 32
    assert many < 4.0 * few, (few, many)


@pytest.mark.parametrize("system", ["rossler_cd", "memristor"])
def test_single_trajectories_that_diverged(engine, system):
    """The one-point form of the other systems."""
    import torch

    values, start, h = {"rossler_cd": ([0.2, 0.2, 0.2, 5.7], [0.0, 0.0, 0.5], 0.01),
                        "memristor": ([1e-5, 1e6], [0.1, 0.5, 0.0], 1e-9)}[system]
    n = 200
    z = lambda t: torch.zeros(n * n, dtype=t, device="cuda")  # noqa: E731
    out = dict(flags=z(torch.int32), avg_peaks=z(torch.float64), avg_intervals=z(torch.float64), counts=z(torch.int32))

    def seconds(samples):
        best = 1e9
        for _ in range(5):
            t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            t[0].record()
            engine.basins_features(system, (samples * 100 + 0.5) * h, n, h, start, [5.0, 20.0, 5.0, 20.0], [0, 1], 0,
                                   1e-3, 0.0, values, preScaller=100, precision="fp32", out=out)
            t[1].record()
            torch.cuda.synchronize()
            best = min(best, t[0].elapsed_time(t[1]))
        assert (out["flags"].cpu().numpy() == 0).all()
        return best

    few, many = seconds(4), seconds(400)
    # one sample against a block of four; a window would run 32
    assert many < 10.0 * few, (few, many)
