"""Basins in FP32, one trajectory per thread and two: with sample counts around
the edges of the windows and of the four samples that are tested on their own,
and with points that leave the bound at the start, inside a window or never,
the features are those of the oracle's peaks in the trajectories of the same
arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYSTEMS = {"lorenz": ([10.0, 24.0, 8 / 3], [0.0, 0.0, 27.0], 0.01, 20.0),
           "rossler": ([0.2, 0.2, 5.7], [0.0, 0.0, 0.5], 0.05, 6.0),
           "chen": ([35.0, 3.0, 28.0], [0.0, 0.0, 20.0], 0.005, 15.0),
           "chameleon": ([0.5, 3.0, 0.0, 2.0, 1.0, 18.0, 1.0], [3.0, 3.0, 0.0], 0.05, 4.0),
           "rossler_cd": ([0.2, 0.2, 0.2, 5.7], [0.0, 0.0, 0.5], 0.01, 6.0),
           "sin3": ([0.5, 0.1, 1.4, 15.552, 2.0], [0.3, -0.2, 0.1], 0.05, 3.0),
           "sin2": ([0.5, 1.0], [0.5, 0.5], 0.05, 3.0)}
N = 9  # 81 points: an odd number


@pytest.mark.parametrize("pre", [1, 3])
@pytest.mark.parametrize("system, pairs", [(s, 0) for s in SYSTEMS] + [(s, 2) for s in ("lorenz", "rossler", "chen")])
def test_windowed_basins_are_the_oracles(engine, oracle, system, pairs, pre):
    values, start, h, reach = SYSTEMS[system]
    axis = -reach + np.arange(N) * (2 * reach / (N - 1))
    x0 = np.tile(np.asarray(start), (N * N, 1))
    x0[:, 0], x0[:, 1] = np.tile(axis, N), np.repeat(axis, N)
    longest = engine.trajectory(system, x0, np.tile(values, (N * N, 1)), h, 110 * pre, precision=engine.FP32)[:, ::pre]
    old = engine.get_tuning(engine.TUNE_SWEEP_PAIRS)
    try:
        engine.set_tuning(engine.TUNE_SWEEP_PAIRS, pairs)
        for wv in (0, 1):
            series = longest[:, :, wv]
            top = np.abs(series).max(axis=1)
            top = top[np.isfinite(top)]  # (some points of rossler_cd leave every bound)
            for maxv in (0.0, float(np.quantile(top, 0.6)), float(np.quantile(np.abs(series[:, 0]), 0.4)) + 1e-3):
                for B in (1, 2, 3, 4, 5, 8, 23, 24, 27, 28, 29, 31, 32, 33, 52, 53, 64, 65, 100):
                    r = engine.basins_features(system, (B + 0.5) * h * pre, N, h, start, [-reach, reach] * 2, [0, 1], wv,
                                               maxv, 0.0, values, pre, precision=engine.FP32)
                    s = series[:, 1:B + 1]
                    inside = (np.abs(s) <= (np.float32(maxv) if maxv else np.finfo(np.float32).max)).all(axis=1)
                    assert np.array_equal(r["flags"] == 0, ~inside), (wv, maxv, B)
                    ok = np.flatnonzero(r["flags"] == 1)
                    counts, pk, iv = oracle.peak_finder(np.ascontiguousarray(series[ok, :B]), h * pre, cap=64)
                    kept = np.maximum(counts, 0)
                    assert np.array_equal(r["counts"][ok], kept), (wv, maxv, B)
                    for i, k in enumerate(ok):
                        m = kept[i]
                        want = (pk[i, :m].mean(), iv[i, :m].mean()) if m else (1000.0, 1000.0)
                        # the sums carry some 48 bits, the mean of the oracle's 53
                        largest = np.abs(pk[i, :m]).max(initial=1.0)
                        assert abs(r["avg_peaks"][k] - want[0]) <= 1e-12 * largest
                        assert abs(r["avg_intervals"][k] - want[1]) <= 1e-12 * max(1.0, want[1])
    finally:
        engine.set_tuning(engine.TUNE_SWEEP_PAIRS, old)
