"""Pairs of trajectories in packed lanes, one of which leaves the bound while it
is on a plateau: the rows of peaks and intervals hold what one point per thread
writes, also in the entries that a diverged point's count leaves unread."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_lane_that_diverges_on_a_plateau(engine):
    """Lorenz with sigma = rho = 0: x stays, y and z turn by about a quarter a
    step with a modulus that beta sets, at sizes where a difference of 1e-13
    (the peak finder's threshold) makes plateaus."""
    import torch

    start = [17.010240918698248, 3.2803374037854804e-15, 2.2567699726773725e-13]
    bound, stays = 7.026300665650835e-13, -3.14
    cap, diverged = 64, 0

    def run(mode, ranges):
        engine.set_tuning(engine.TUNE_SWEEP_PAIRS, mode)
        z = lambda shape, t: torch.zeros(shape, dtype=t, device="cuda")  # noqa: E731
        out = dict(counts=z(2, torch.int32), flags=z(2, torch.int32), first=z(2, torch.float64),
                   peaks=z((2, cap), torch.float64), intervals=z((2, cap), torch.float64))
        engine.bifurcation1d("lorenz", 40.0, 2, 0.1, start, ranges, [2], 1, bound, 0.0, [0.0, 0.0, 0.0],
                             peakCapacity=cap, precision="fp32", out=out)
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in out.items()}

    try:
        for leaves in np.linspace(-7.0, -5.7, 40):
            for ranges in ([leaves, stays], [stays, leaves]):
                single, pair = run(0, ranges), run(2, ranges)
                diverged += sorted(single["flags"]) == [-1, 0]  # (steps of 1e-13 count as a fixed point)
                for k in single:
                    assert np.array_equal(single[k], pair[k]), (k, ranges)
    finally:
        engine.set_tuning(engine.TUNE_SWEEP_PAIRS, 1)
    assert diverged > 40
