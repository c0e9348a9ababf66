"""The windowed peak detector of the FP32 sweeps (PeakWindow, chaoslibrary_gb300/
csrc/peaks.h) on the host: on series full of ties, plateaus and steps around
the 1e-13 threshold it finds, window by window, exactly the peaks that the
one-at-a-time detector (PeakStream) finds, for every window length and for a
last window cut short."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]

CHECKER = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "peaks.h"
struct Peak { float v; int t; };
// argv: series file, series, length, window; exit 0 when both detectors agree on every series, 2 when none found a peak
int main(int, char** argv) {
    const int n = atoi(argv[2]), len = atoi(argv[3]), win = atoi(argv[4]);
    std::vector<float> d((size_t)n * len);
    FILE* f = fopen(argv[1], "rb");
    if (!f || fread(d.data(), sizeof(float), d.size(), f) != d.size()) return 1;
    fclose(f);
    size_t found = 0;
    for (int s = 0; s < n; ++s) {
        const float* x = d.data() + (size_t)s * len;
        std::vector<Peak> a, b;
        chaos::PeakStream<float> ps;
        ps.init();
        for (int k = 0; k < len; ++k) {
            float v;
            int t;
            if (ps.push(x[k], v, t)) a.push_back({v, t});
        }
        chaos::PeakWindow pw;
        pw.init();
        unsigned up = 0;
        for (int k0 = 0; k0 < len; k0 += win) {
            const int m = len - k0 < win ? len - k0 : win;
            auto at = [&](int j) { return k0 + j < 0 ? 0.f : x[k0 + j]; };
            auto peak = [&](float v, int t) { b.push_back({v, t}); };
            unsigned mask = 0;
            for (int j = 0; j < m; ++j) mask = (mask << 1) | (at(j) > at(j - 1));
            unsigned cand = chaos::PeakWindow::candidates(mask, up, m);
            up = mask & 1;
            if (pw.i0 >= 0) pw.walk(k0, 0, m, at, peak);
            while (cand) {
                const int j = chaos::PeakWindow::next(cand, m);
                pw.judge(k0, j, m, at, peak);
            }
        }
        if (a.size() != b.size()) return 3;
        for (size_t i = 0; i < a.size(); ++i)
            if (a[i].v != b[i].v || a[i].t != b[i].t) return 4;
        found += a.size();
    }
    return found > 0 ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("window")
    src = d / "peak_window_check.cpp"
    src.write_text(CHECKER)
    exe = d / "peak_window_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'chaoslibrary_gb300' / 'csrc'}",
                    str(src), "-o", str(exe)], check=True)

    def run(data, window):
        data = np.ascontiguousarray(data, np.float32)
        data.tofile(d / "in.bin")
        return subprocess.run([str(exe), str(d / "in.bin"), str(data.shape[0]), str(data.shape[1]),
                               str(window)]).returncode

    return run


def _series(rng, kind, n, ln):
    if kind == "levels":  # ties, runs of equal samples
        d = rng.integers(-2, 3, size=(n, ln)) * 0.25
        d[: n // 4] = np.repeat(d[: n // 4, ::5], 5, axis=1)[:, :ln]
        return d
    if kind == "threshold":  # steps just above and below 1e-13, where float resolves them; both signs of zero
        d = rng.choice([0.0, -0.0, 1e-12, 1.1e-12, 1.15e-12, 1.2e-12, -1e-12], size=(n, ln))
        d[: n // 4] = np.repeat(d[: n // 4, ::7], 7, axis=1)[:, :ln]
        return d
    t = np.arange(ln)  # smooth orbits that settle: long monotone stretches, then equal samples for good
    w, a = rng.uniform(0.05, 2.5, (n, 1)), rng.uniform(0.0, 0.2, (n, 1))
    return np.exp(-a * t) * np.sin(w * t)


@pytest.mark.parametrize("kind", ["levels", "threshold", "settling"])
@pytest.mark.parametrize("window", [1, 2, 3, 15, 16, 31, 32])
def test_windows_find_the_streams_peaks(checker, kind, window):
    rng = np.random.default_rng(11)
    for ln in (1, 2, 3, 5, 16, 33, 257):
        rc = checker(_series(rng, kind, 200, ln), window)
        assert rc == 0 or (rc == 2 and ln < 5), (kind, window, ln, rc)
