"""FP32 and float-float LLE maps and the FP32 spectrum run two points per
thread, and one row of blocks one point per thread where the points fill an
odd number of rows: at sizes with no pair block, no single block and both, and
with an odd last point, every point has the bits of the other form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAPS = {"lorenz": ([10.0, 28.0, 8 / 3], [1.0, 1.0, 1.0], [1, 0], [20.0, 200.0, 5.0, 15.0]),
        "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 1.0], [0, 2], [0.1, 0.4, 2.0, 10.0]),
        "chen": ([35.0, 3.0, 28.0], [-10.0, 0.0, 37.0], [2, 0], [20.0, 30.0, 30.0, 40.0])}


@pytest.mark.parametrize("system", sorted(MAPS))
@pytest.mark.parametrize("n", [1, 12, 139, 197, 203, 241, 279])  # 1, 1, 1, 2, 3, 3 and 5 rows on 152 SMs
def test_lle_single_and_paired_rows(engine, system, n):
    values, ic, mut, rg = MAPS[system]
    kw = dict(tMax=4.0, NT=0.2, nPts=n, h=0.01, eps=1e-8, initialConditions=ic, ranges=rg, indicesOfMutVars=mut,
              transientTime=2.0, values=values)
    for precision, knob, forms in (("fp32", engine.TUNE_LLE_F32_VARIANT, (0, 2, 12)),
                                   ("ff32", engine.TUNE_FF_PAIRS, (1, 0))):
        old = engine.get_tuning(engine.TUNE_FF_PAIRS)
        res = []
        try:
            for v in forms:
                engine.set_tuning(knob, v)
                res.append(engine.lle2d(system, precision=precision, **kw))
        finally:
            engine.set_tuning(engine.TUNE_LLE_F32_VARIANT, 0)
            engine.set_tuning(engine.TUNE_FF_PAIRS, old)
        for r in res[1:]:
            assert np.array_equal(res[0], r, equal_nan=True), (precision, n)


@pytest.mark.parametrize("system", sorted(MAPS))
def test_spectrum_single_and_paired_rows(engine, system):
    values, ic, mut, rg = MAPS[system]
    kw = dict(tMax=3.0, NT=0.1, h=0.01, eps=1e-8, initialConditions=ic, indicesOfMutVars=mut, transientTime=1.0,
              values=values, precision="fp32")
    n = 40001  # three rows on 152 SMs: one single, then pairs, the last thread with one point
    big = engine.lyapunov_spectrum(system, 1, nPts=n, ranges=rg[:2], **kw)
    step = (rg[1] - rg[0]) / (n - 1)
    for k in (0, 19455, 19456, 19457, 30001, n - 2, n - 1):
        one = engine.lyapunov_spectrum(system, 1, nPts=2, ranges=[rg[0] + k * step, rg[0] + k * step + 1e-3], **kw)
        assert np.array_equal(one[0], big[k]), k
