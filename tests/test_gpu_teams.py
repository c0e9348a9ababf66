"""Small FP64 sweeps of the RK4 systems run a trajectory on a team of three
lanes, ten teams a warp (an LLE point's orbit and twin in one team or in two):
around whole and partly filled warps, for every recorded component, with
points that leave the bound in the transient or while they record, they give
the oracle's results bit for bit, and the LLE maps those of the kernel that
runs a point per thread."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYSTEMS = {"lorenz": ([10.0, 28.0, 8 / 3], [0.1, -0.1, 0.1], 1, [0.5, 200.0]),  # fixed points among them
           "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 1.0], 2, [2.0, 10.0]),
           "chen": ([35.0, 3.0, 28.0], [-10.0, 0.0, 37.0], 2, [20.0, 30.0])}
SYSTEM_ID = {"lorenz": 0, "rossler": 1, "chen": 2}


@pytest.mark.parametrize("system", sorted(SYSTEMS))
@pytest.mark.parametrize("wv", [0, 1, 2])
@pytest.mark.parametrize("n", [2, 9, 10, 11, 31, 67])
def test_bifurcation_teams_are_the_oracle(engine, oracle, system, wv, n):
    values, ic, mi, rg = SYSTEMS[system]
    for tMax, trans, maxv in ((0.32, 0.0, 1e4), (0.33, 0.09, 0.0), (6.4, 1.0, 1e4), (4.0, 2.0, 25.0)):
        kw = dict(tMax=tMax, nPts=n, h=0.01, ranges=rg, maxValue=maxv, transientTime=trans, values=values)
        r = engine.bifurcation1d(system, initialConditions=ic, indicesOfMutVars=[mi], writableVar=wv, peakCapacity=64,
                                 **kw)
        o = oracle.bifurcation(SYSTEM_ID[system], dim=1, cap=64, ic=ic, mut=[mi], wv=wv, **kw)
        assert np.array_equal(r["counts"], o["counts"]) and np.array_equal(r["flags"], o["flags"])
        for k, c in enumerate(r["counts"]):
            if c > 0:
                assert np.array_equal(r["peaks"][k, :c], o["peaks"][k, :c])
                assert np.array_equal(r["intervals"][k, :c], o["intervals"][k, :c])


@pytest.mark.parametrize("system", sorted(SYSTEMS))
@pytest.mark.parametrize("pre", [1, 3])
def test_basins_teams_are_the_oracle(engine, oracle, system, pre):
    values, _, _, _ = SYSTEMS[system]
    for n, wv, maxv in ((2, 0, 1e8), (5, 1, 1e8), (11, 2, 30.0)):
        kw = dict(tMax=9.7, nPts=n, h=0.01, ranges=[-30.0, 30.0, -30.0, 30.0], maxValue=maxv, transientTime=2.0,
                  values=values, preScaller=pre)
        ic = [0.0, 0.0, 20.0]
        r = engine.basins_features(system, initialConditions=ic, indicesOfMutVars=[0, 1], writableVar=wv, **kw)
        o = oracle.basins_features(SYSTEM_ID[system], ic=ic, mut=[0, 1], wv=wv, **kw)
        for k in ("flags", "avg_peaks", "avg_intervals", "counts"):
            assert np.array_equal(r[k], o[k]), (k, n)


@pytest.mark.parametrize("system", sorted(SYSTEMS))
@pytest.mark.parametrize("twin", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 80])  # 80^2 points: above 40 per SM, orbit and twin in one team
def test_lle_teams_are_the_point_kernel(engine, system, twin, n):
    values, ic, mi, rg = SYSTEMS[system]
    rg = [max(rg[0], 2.0), rg[1]]
    other = (mi + 1) % 3
    ranges = [rg[0], rg[1], values[other], values[other] + 0.25]
    eps, h, trans = 1e-8, 0.01, 1.37
    old = engine.get_tuning(engine.TUNE_LLE_TWIN)
    try:
        engine.set_tuning(engine.TUNE_LLE_TWIN, twin)
        got = engine.lle2d(system, 3.0, 0.07, n, h, eps, ic, ranges, [mi, other], trans, values)
    finally:
        engine.set_tuning(engine.TUNE_LLE_TWIN, old)
    k = np.arange(n)
    step = [(ranges[1] - ranges[0]) / (n - 1), (ranges[3] - ranges[2]) / (n - 1)] if n > 1 else [0.0, 0.0]
    a = np.tile(values, (n * n, 1))
    a[:, mi] = np.tile(ranges[0] + k * step[0], n)
    a[:, other] = np.repeat(ranges[2] + k * step[1], n)
    x = engine.trajectory(system, np.tile(ic, (n * n, 1)), a, h, int(trans / h))[:, -1]
    q = x.copy()
    if twin:  # every component rounded to float, eps added to the first in float
        q = x.astype(np.float32).astype(np.float64)
        q[:, 0] = (q[:, 0] + float(np.float32(eps))).astype(np.float32)
    else:
        q[:, 0] += eps
    want = engine.lle_from_states(system, np.concatenate([x, a, q], axis=1), 3.0, 0.07, h, eps)
    assert np.array_equal(got, want, equal_nan=True)
