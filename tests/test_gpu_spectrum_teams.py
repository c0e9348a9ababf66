"""FP64 spectra of the RK4 systems on teams of three lanes -- the four
trajectories of a point in a team each (up to 28 points per SM) or in one (up to
76) -- against the kernel that runs a point per thread, bit for bit: single
points, ragged warps, both edges of the rules, odd numbers of steps a block,
no transient, and a twin distance that vanishes beside the state, so that
norms, projections and their denominators are zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SYSTEMS = {"lorenz": ([10.0, 28.0, 8 / 3], [1.0, 1.0, 1.0], 1, 20.0, 1 / 64),
           "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 1.0], 2, 2.0, 1 / 2048),
           "chen": ([35.0, 3.0, 28.0], [-10.0, 0.0, 37.0], 2, 20.0, 1 / 2048)}


@pytest.mark.parametrize("system", sorted(SYSTEMS))
@pytest.mark.parametrize("NT, eps, transient", [(0.07, 1e-8, 0.5), (0.1, 1e-20, 0.0), (0.01, 1e-3, 0.11)])
def test_spectrum_teams_are_the_point_kernel(engine, system, NT, eps, transient):
    import torch

    values, ic, mut, start, step = SYSTEMS[system]
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def spectrum(n):  # the first n points of one grid, whose step is exact
        r = engine.lyapunov_spectrum(system, 1, 0.7, NT, n, 0.01, eps, ic, [start, start + (n - 1) * step], [mut],
                                     transient, values)
        return np.asarray(r).reshape(n, 3)

    full = spectrum(100 * sms)
    for n in (2, 3, 5, 28 * sms - 1, 28 * sms, 28 * sms + 1, 28 * sms + 17, 76 * sms, 76 * sms + 1):
        assert np.array_equal(spectrum(n).view(np.int64), full[:n].view(np.int64)), n
