"""The FP32 sweeps judge their recorded samples in windows (32 for one
trajectory per thread, 24 for two): with sample counts around the windows'
edges, every recorded component and points that leave the bound inside a
window, the peaks are those the oracle's peak finder sees in the trajectories
of the same arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYSTEMS = {"lorenz": ([10.0, 28.0, 8 / 3], [0.1, 0.1, 0.1], 1, [20.0, 200.0]),
           "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 1.0], 2, [2.0, 10.0])}
N, H = 67, 0.05  # a coarse step: peaks every few samples


@pytest.mark.parametrize("pairs", [0, 2])
@pytest.mark.parametrize("system", sorted(SYSTEMS))
@pytest.mark.parametrize("wv", [0, 1, 2])
def test_windowed_peaks_are_the_oracles(engine, oracle, system, pairs, wv):
    values, ic, mi, rg = SYSTEMS[system]
    h = H if system == "rossler" else H / 5
    a = np.tile(values, (N, 1))
    a[:, mi] = rg[0] + np.arange(N) * ((rg[1] - rg[0]) / (N - 1))
    longest = engine.trajectory(system, np.tile(ic, (N, 1)), a, h, 400, precision=engine.FP32)[:, :, wv]
    bound = float(np.quantile(np.abs(longest).max(axis=1), 0.6))  # two of five points leave it somewhere
    old = engine.get_tuning(engine.TUNE_SWEEP_PAIRS)
    try:
        engine.set_tuning(engine.TUNE_SWEEP_PAIRS, pairs)
        for B in (1, 2, 3, 23, 24, 25, 31, 32, 33, 48, 49, 64, 65, 96, 97, 400):
            for maxv in (0.0, bound):
                r = engine.bifurcation1d(system, (B + 0.5) * h, N, h, ic, rg, [mi], wv, maxv, 0.0, values,
                                         peakCapacity=400, precision=engine.FP32)
                counts, pk, iv = oracle.peak_finder(longest[:, :B], h, cap=400)
                inside = np.abs(longest[:, 1:B + 1]).max(axis=1) <= np.float32(maxv) if maxv else np.ones(N, bool)
                assert np.array_equal(r["flags"] == 0, ~inside), (B, maxv)
                ok = r["flags"] == 1
                assert np.array_equal(r["counts"][ok], counts[ok]), (B, maxv)
                assert np.array_equal(r["first"], longest[:, 0])
                for k in np.flatnonzero(ok):
                    c = counts[k]
                    assert np.array_equal(r["peaks"][k, :c], pk[k, :c]), (B, maxv, k)
                    assert np.array_equal(r["intervals"][k, :c], iv[k, :c]), (B, maxv, k)
    finally:
        engine.set_tuning(engine.TUNE_SWEEP_PAIRS, old)
