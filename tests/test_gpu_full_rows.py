"""FP32 and float-float maps of whole rows of 128 points per SM, or a few blocks
short of that: the same bits in slices and in one launch, and three full rows
of a spectrum take less than four."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYSTEMS = {"lorenz": ([10.0, 28.0, 8 / 3], [1.0, 1.0, 1.0], [1], [20.0, 200.0]),
           "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 1.0], [2], [2.0, 10.0]),
           "chen": ([35.0, 3.0, 28.0], [-10.0, 0.0, 37.0], [2], [20.0, 30.0])}


def _runner(engine, system, kind, precision, n, tMax):
    import torch

    values, ic, mut, rg = SYSTEMS[system]
    call = engine.lle_sweep if kind == "lle" else engine.lyapunov_spectrum
    out = torch.zeros(n * (1 if kind == "lle" else 3), dtype=torch.float64, device="cuda")
    return out, lambda: call(system, 1, tMax, 0.1, n, 0.01, 1e-8, ic, rg, mut, 2.0, values, precision=precision, out=out)


def _row():
    import torch

    return 128 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("system", sorted(SYSTEMS))
@pytest.mark.parametrize("kind, precision", [("lle", "fp32"), ("lle", "ff32"), ("spectrum", "fp32")])
@pytest.mark.parametrize("rows", [2, 3, 5, 7])
def test_full_rows(engine, system, kind, precision, rows):
    import torch

    for n in (rows * _row(), rows * _row() - 1, (rows * _row()) - 13 * 256 + 1):
        out, run = _runner(engine, system, kind, precision, n, 20.0)
        run()
        torch.cuda.synchronize()
        direct = out.cpu().numpy()
        out.zero_()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(direct.view(np.int64), out.cpu().numpy().view(np.int64)), n
        # the ends of the map against a map of its own, one point per thread
        few, alone = _runner(engine, system, kind, precision, 2, 20.0)
        alone()
        torch.cuda.synchronize()
        w = 1 if kind == "lle" else 3
        assert np.array_equal(few.cpu().numpy().view(np.int64), np.concatenate([direct[:w], direct[-w:]]).view(np.int64))


@pytest.mark.parametrize("system", sorted(SYSTEMS))
def test_three_rows_take_less_than_four(engine, system):
    import torch

    def ms(rows):
        _, run = _runner(engine, system, "spectrum", "fp32", rows * _row(), 60.0)
        run()
        best = 1e9
        for _ in range(7):
            t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            t[0].record()
            run()
            t[1].record()
            torch.cuda.synchronize()
            best = min(best, t[0].elapsed_time(t[1]))
        return best

    three, four = ms(3), ms(4)
    assert three < 0.9 * four, (three, four)
