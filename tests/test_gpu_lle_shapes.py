"""The FP32 LLE map's launch shapes: reading the variant and setting it again
changes nothing, and a shape that the tuner found on large maps is not used for
the sizes that run in slices or in mixed blocks."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(engine, n):
    import torch

    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    before = engine.launch_count()
    engine.lle_sweep("lorenz", 1, 60.0, 0.1, n, 0.01, 1e-8, [1.0, 1.0, 1.0], [20.0, 200.0], [1], 5.0,
                     [10.0, 28.0, 8 / 3], precision="fp32", out=out)
    torch.cuda.synchronize()
    return engine.launch_count() - before, out.cpu().numpy()


def test_reading_and_setting_the_variant(engine):
    import torch

    n = 128 * torch.cuda.get_device_properties(0).multi_processor_count + 131
    launches, values = _map(engine, n)
    assert launches > 1  # in slices
    knob = engine.TUNE_LLE_F32_VARIANT
    try:
        assert engine.get_tuning(knob) == 0
        engine.set_tuning(knob, engine.get_tuning(knob))
        again, same = _map(engine, n)
        assert again == launches and np.array_equal(values, same)
        for v in (2, 12, 16):
            engine.set_tuning(knob, v)
            assert engine.get_tuning(knob) == v
            assert _map(engine, n)[0] == 1
    finally:
        engine.set_tuning(knob, 0)


@pytest.mark.parametrize("shape", [2 * 1024 + 64, 12 * 1024 + 128])
def test_a_tuned_shape_leaves_smaller_maps(engine, shape):
    import torch

    row = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    install = getattr(engine.lib(), "_ZN5chaos16set_launch_shapeEiii")  # what chaos_autotune calls
    install.argtypes, install.restype = [ctypes.c_int] * 3, ctypes.c_int
    small, large = row + 131, 23 * row
    rule = [_map(engine, n) for n in (small, large)]
    try:
        assert install(2, 0, shape) == 0
        tuned = [_map(engine, n) for n in (small, large)]
    finally:
        engine.set_tuning(engine.TUNE_SHAPES, 0)
    assert tuned[0][0] == rule[0][0] > 1
    for (_, a), (_, b) in zip(rule, tuned):
        assert np.array_equal(a, b)
