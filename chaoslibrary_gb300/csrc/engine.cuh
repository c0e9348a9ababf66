// Device-side building blocks of the sweep engine: per-launch parameter
// blocks, the streaming peak detector, the divergence / fixed-point tests and
// the per-point work functions of the three analyses. Included by the FP64
// and the FP32 kernel translation units, which instantiate the templates for
// their arithmetic type.
//
// Layout rule for every kernel here: one CUDA thread owns one trajectory (two in
// the packed FP32 forms; in small FP64 sweeps three lanes share one, team.cuh).
// State and parameters live in registers, with the FP64 peak detector; the FP32
// sweeps keep a window of samples and their detectors in shared memory. The
// trajectory itself never reaches HBM, but for the state of points whose
// horizon runs in slices. What a point writes to HBM is its result row (a few
// scalars, plus its peak list for the bifurcation sweeps).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "launch.h"
#include "order_keys.h"
#include "peaks.h"
#include "systems.h"
#include "ff.h"

namespace chaos {

template <int S> struct Traits {
    static constexpr int NX = (S == SYS_SIN2) ? 2 : 3;
    static constexpr int NA = (S == SYS_CHAMELEON) ? 7 : (S == SYS_ROSSLER_CD) ? 4 : (S == SYS_SIN3) ? 5
                            : (S == SYS_SIN2 || S == SYS_MEMRISTOR) ? 2 : 3;
};
#if defined(CHAOS_USER_SYSTEM)
template <> struct Traits<SYS_USER> {
    static constexpr int NX = CHAOS_USER_NX;
    static constexpr int NA = CHAOS_USER_NA;
};
#endif

// Swept value of grid dimension d for linear point index p (the reference's
// getValueByIdx, bifurcationCUDA.cu:400-419 / basinsCUDA.cu:185-189):
// start + n*scale with n = (p / nPts^d) % nPts, multiply and add rounded apart
// (the source as written), or as one FMA when g.fused (the reference's own
// GPU build: nvcc contracts the expression by default).
__device__ __forceinline__ double grid_value(const GridSpec& g, long long p, int d) {
    long long q = p;
    if (d == 1) q /= g.nPts;
    const long long n = q % g.nPts;
    if (g.table[d]) return g.table[d][n];
    return g.fused ? __fma_rn((double)n, g.scale[d], g.start[d]) : __dadd_rn(g.start[d], __dmul_rn((double)n, g.scale[d]));
}

// The maxValue test of both loops, (double)fabsf((float)v) > maxValue, for a
// double v on the integer pipe (this GPU's FP64 pipe is its bottleneck in the
// FP64 sweeps): with b the bits of |v| (not NaN), it holds exactly when
// b > maxBits, or b == maxBits and maxTie (the host derives maxBits from the
// rounding boundary of float(v) at maxValue, see fill_sweep).
__device__ __forceinline__ bool max_exceeded(unsigned long long b, const SweepParams& P) {
    return b > P.maxBits || (b == P.maxBits && P.maxTie);
}

// Divergence test of the bifurcation loop (bifurcationCUDA.cu:445-453):
// v != v || v == v + 1.0  <=>  !(|v| < 2^53); then |(float)v| > maxValue.
template <class T> __device__ __forceinline__ bool bif_diverged(T v, const SweepParams& P);
template <> __device__ __forceinline__ bool bif_diverged<double>(double v, const SweepParams& P) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    if (b >= 0x4340000000000000ull) return true;  // |v| >= 2^53, infinite or NaN
    return P.checkMax && max_exceeded(b, P);
}
// The same test for a float v, as one compare against a limit that does not
// change in the loop: !(|v| < 2^53) || (checkMax && |v| > maxValueF) holds
// exactly when !(|v| <= lim), lim = min(maxValueF, 2^53 - 2^29) with checkMax,
// else 2^53 - 2^29 (the largest float below 2^53); NaN fails every compare.
template <> __device__ __forceinline__ bool bif_diverged<float>(float v, const SweepParams& P) {
    constexpr float kBelow2p53 = 9007198717870080.0f;
    const float lim = P.checkMax ? fminf(P.maxValueF, kBelow2p53) : kBelow2p53;
    return !(fabsf(v) <= lim);
}
// Divergence test of the basins loop (basinsCUDA.cu:350-361): isnan || isinf, then maxValue.
template <class T> __device__ __forceinline__ bool basins_diverged(T v, const SweepParams& P);
template <> __device__ __forceinline__ bool basins_diverged<double>(double v, const SweepParams& P) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    if (b > 0x7fefffffffffffffull) return true;  // NaN or +-inf
    return P.checkMax && max_exceeded(b, P);
}
// As one compare: a limit that is negative or below the largest float decides
// alone, a NaN limit (never exceeded) leaves the largest float.
template <> __device__ __forceinline__ bool basins_diverged<float>(float v, const SweepParams& P) {
    constexpr float kMax = 3.4028234663852886e38f;
    const float lim = P.checkMax ? fminf(P.maxValueF, kMax) : kMax;
    return !(fabsf(v) <= lim);
}

// The sample tests and the streaming peak detector (PeakStream) live in
// peaks.h, which the host compiles too.

// x[wv] for a run-time wv without indexing the register array (which would
// move the whole state to local memory).
template <int NX, class T> __device__ __forceinline__ T pick(const T* x, int wv) {
    T v = x[0];
#pragma unroll
    for (int j = 1; j < NX; ++j)
        if (j == wv) v = x[j];
    return v;
}

// The recorded component of a sweep: known at compile time (W >= 0), or at run
// time. The FP32 sweeps of the RK4 systems and of Chameleon run their loops
// with the component known: picking it costs two selects a sample and
// trajectory otherwise, which the packed loops' ALU pipe feels (700,001
// Rossler points 18.6 -> 17.7 ms, 1,000 Lorenz points 0.90 -> 0.84 ms).
template <int W> struct Component {
    static constexpr int kIndex = W;
    int wv;
    template <int NX, class T> __device__ __forceinline__ T of(const T* x) const {
        if constexpr (W >= 0) return x[W < NX ? W : 0];
        else return pick<NX>(x, wv);
    }
};
template <int S, class T> struct KnownComponent {
    static constexpr bool value = std::is_same<T, float>::value && (S <= SYS_CHEN_RK4 || S == SYS_CHAMELEON);
};
// f(component) for the component wv of a sweep: one copy of f per component of
// a system with KnownComponent (three components), else one for all. The
// single-sweep kernels choose on the host, a kernel per component (three
// copies in one kernel share its registers and its schedule: 1,000 Lorenz
// points took 1.17 ms in that form), a batch's kernels on the device, chunk by chunk.
template <bool Known, class Fn> __host__ __device__ __forceinline__ void with_component(int wv, Fn&& f) {
    if constexpr (Known) {
        if (wv == 0) f(Component<0>{0});
        else if (wv == 1) f(Component<1>{1});
        else f(Component<2>{2});
    } else {
        f(Component<-1>{wv});
    }
}

// Loads state and parameters of point p of a sweep (mutated parameters or
// mutated initial-condition components, per P.mutateState).
template <int S, class T> __device__ __forceinline__ void load_point(const SweepParams& P, long long p, T* x, T* a) {
    constexpr int NX = Traits<S>::NX, NA = Traits<S>::NA;
    double v0 = 0.0, v1 = 0.0;
    v0 = grid_value(P.grid, p, 0);
    if (P.dim > 1) v1 = grid_value(P.grid, p, 1);
#pragma unroll
    for (int i = 0; i < NX; ++i) {
        double v = P.ic[i];
        if (P.mutateState) {  // dimension 1 is written last, as in the reference loop
            if (i == P.mut[0]) v = v0;
            if (P.dim > 1 && i == P.mut[1]) v = v1;
        }
        x[i] = (T)v;
    }
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        double v = P.values[i];
        if (!P.mutateState) {
            if (i == P.mut[0]) v = v0;
            if (P.dim > 1 && i == P.mut[1]) v = v1;
        }
        a[i] = (T)v;
    }
}

// Fixed-point test of the bifurcation loop: sqrtf(fabsf(sum)) < 1e-9 in float.
template <int NX, class T> __device__ __forceinline__ bool bif_fixed(const T* x, const T* xp) {
    T s = T(0);
#pragma unroll
    for (int j = 0; j < NX; ++j) s = s + (x[j] - xp[j]) * (x[j] - xp[j]);
    return (double)sqrtf(fabsf((float)s)) < 1e-9;
}
// Fixed-point test of the basins loop: sqrt(abs(sum)) < 1e-9 in FP64.
template <int NX, class T> __device__ __forceinline__ bool basins_fixed(const T* x, const T* xp) {
    T s = T(0);
#pragma unroll
    for (int j = 0; j < NX; ++j) s = s + (x[j] - xp[j]) * (x[j] - xp[j]);
    return sqrt(fabs((double)s)) < 1e-9;
}

// Steps per block of the bifurcation transients' block form.
constexpr int kTransientBlock = 8;

// Steps laid out one after the other in the FP32 loops: transient steps before a
// test, and samples of a window in a row. sin3 and the memristor have long steps
// with branches of their own (the slow ranges of the sines and exponentials), and
// copies of them fetch and wait: sin3, 40 time units, 1,000 points 2.4 -> 1.7 ms,
// 400,000 14.7 -> 12.4; its basins 30^2 0.97 -> 0.86; memristor 1,000 points 2.79 ->
// 2.76 ms, 400,000 21.0 -> 18.4 (one sample in a row 2.98 and 17.7: left at four).
// sin2 basins of 400^2 points, several steps a sample, 1.14 -> 1.12 ms with two in
// a row, but 1.08 -> 1.13 with one step a sample.
template <int S> struct Straight {
    static constexpr int kTransient = S == SYS_SIN3 || S == SYS_MEMRISTOR ? 1 : kTransientBlock;
    static constexpr int kSamples = S == SYS_SIN3 ? 1 : 4;  // of one step each
    static constexpr int kLongSamples = S == SYS_SIN2 ? 2 : kSamples;
};

// The FP32 recorded loops judge their samples in windows (PeakWindow,
// peaks.h). A thread runs L trajectories (1, or 2 in packed lanes); what it
// needs once a window lives in shared memory, so that the step loop keeps its
// registers: the samples of the window and the two before it, the detectors
// and a basins point's sums. A thread's samples are one column whose length
// is odd in units of a bank row's step (L words), so a warp's stores of one
// sample are free of bank conflicts.
// 32 samples a window for one trajectory, 24 for two: the longer, the rarer
// the judging (700,001 Rossler points 18.3 ms with 16 in two lanes, 18.1 with
// 24), but 24 already leave room for only six blocks of 128 threads per SM.
template <int L> struct Window {
    static constexpr int K = L == 1 ? 32 : 24;  // samples
    static constexpr int kColumn = (K + 3) * L;  // floats of a thread's column: 2 + K samples, 1 unused
    static constexpr size_t kDetectors = sizeof(int4) * L, kSums = sizeof(float4) * L;
    static constexpr size_t bytes(int block) { return (kDetectors + kSums + kColumn * sizeof(float)) * block; }

    int4* det;     // [L][blockDim.x]
    float4* sum;   // [L][blockDim.x]
    float* col;    // this thread's column
    __device__ __forceinline__ Window() {
        extern __shared__ int4 window_smem[];
        det = window_smem + threadIdx.x;
        sum = reinterpret_cast<float4*>(window_smem + L * blockDim.x) + threadIdx.x;
        col = reinterpret_cast<float*>(window_smem + 2 * L * blockDim.x) + kColumn * threadIdx.x;
    }
    __device__ __forceinline__ float& at(int l, int j) const { return col[(j + 2) * L + l]; }  // -2 <= j < K
    __device__ __forceinline__ void put(int j, float v) const { col[j + 2] = v; }
    __device__ __forceinline__ void put(int j, float2 v) const { reinterpret_cast<float2*>(col)[j + 2] = v; }
    __device__ __forceinline__ PeakWindow detector(int l) const {
        const int4 d = det[l * blockDim.x];
        return PeakWindow{d.x, d.y, d.z, d.w};
    }
    __device__ __forceinline__ void keep(int l, const PeakWindow& d) const {
        det[l * blockDim.x] = make_int4(d.nc, d.i0, d.n, d.tprev);
    }

    // Judges the candidates of one window that starts at sample index k: the
    // lanes' candidates one after the other in one loop, so that a warp goes
    // round as often as its busiest thread has candidates. open: bit l set
    // while lane l's detector is on a plateau; moved: those of them whose
    // window is not all one value (an orbit that has come to rest leaves its
    // plateau open for good, and walking along it would cost more than its
    // steps: 1,000 Lorenz points with such orbits among them 1.33 -> 0.93 ms).
    // on_peak(l, detector, val, t) sees the detector before the peak is counted.
    template <class OnPeak>
    __device__ __forceinline__ void judge(int k, unsigned c0, unsigned c1, int m0, int m1, unsigned moved,
                                          unsigned& open, OnPeak&& on_peak) const {
        PeakWindow d0 = detector(0), d1 = d0;
        if (L == 2) d1 = detector(1);
        auto run = [&](PeakWindow& d, int l, int j, int m) {  // j < 0: a plateau from the window before
            auto a = [&](int i) { return at(l, i); };
            auto peak = [&](float val, int t) {
                on_peak(l, d, val, t);
                d.tprev = t;
                ++d.n;
            };
            if (j < 0) d.walk(k, 0, m, a, peak);
            else d.judge(k, j, m, a, peak);
        };
        if (moved & 1u) run(d0, 0, -1, m0);
        if (L == 2 && (moved & 2u)) run(d1, 1, -1, m1);
        while ((c0 | c1) != 0u) {
            if (L == 1) {
                const int j = PeakWindow::next(c0, m0);
                run(d0, 0, j, m0);
            } else {
                const int l = c0 == 0u ? 1 : 0, m = l ? m1 : m0;
                unsigned c = l ? c1 : c0;
                const int j = PeakWindow::next(c, m);
                if (l) c1 = c;
                else c0 = c;
                PeakWindow d = l ? d1 : d0;
                run(d, l, j, m);
                if (l) d1 = d;
                else d0 = d;
            }
        }
        open = (d0.i0 >= 0 ? 1u : 0u) | (L == 2 && d1.i0 >= 0 ? 2u : 0u);
        keep(0, d0);
        if (L == 2) keep(1, d1);
    }
};

// The recorded loop of one FP32 trajectory: B samples x[wv], one before each
// advance(); diverged(v) ends the point (returned as 0, otherwise 1); xp
// receives the state before the last advance of a point that did not diverge,
// last the last sample and n the detected peaks. on_peak(l, detector, val, t)
// for every detected peak, in order.
//
// What bounds it is issue slots (large sweeps) or one warp's chain (small
// ones), so a sample costs two compares, a predicated bit and a shared store
// beside its step, and the peak rules run once a window for the whole warp.
// Judging blocks of 4 samples instead (a gate of two compares and two selects
// a sample) sent nearly every block of a chaotic sweep through the
// transitions sample by sample, since one of 32 orbits always had a peak in
// it. Measured against that, 20,000 steps: 1,000 Lorenz points (then with the
// detector as selects) 1.83 -> 0.88 ms, 700,001 Rossler points 19.9 -> 18.1 ms.
//
// Stop: a window ends after the four samples among which the orbit diverged. In
// maps with many such points the rest of the window is time lost (basins of 40
// time units, 5 steps a sample: rossler_cd 400^2 0.370 -> 0.303 ms, memristor
// 900^2 12.9 -> 11.7); the basins of the RK4 systems and of Chameleon with one
// step a sample go without, where the test costs up to 5 % (Rossler 400^2 0.757
// -> 0.799 ms) and a window at most some 2 us. Samples: of a window in a row.
template <int NX, bool Stop, int Samples, int W, class Advance, class Diverged, class OnPeak>
__device__ __forceinline__ int record_windows(int B, float* x, float* xp, Component<W> wc, const Window<1>& w, float& last,
                                              int& n, Advance&& advance, Diverged&& diverged, OnPeak&& on_peak) {
    constexpr int K = Window<1>::K;
    PeakWindow d;
    d.init();
    w.keep(0, d);
    w.put(-2, 0.f);
    w.put(-1, 0.f);
    float v = wc.template of<NX>(x), p = 0.f;  // the recorded sample, carried from one step to the next
    unsigned up = 0, open = 0;
    int i = 0;
    bool dv = false;
    for (; i + K < B; i += K) {
        unsigned mask = 0;
        int q = 0;
#pragma unroll 1
        for (; q < K && !(Stop && dv); q += 4) {
            mask <<= 4;
#pragma unroll (Samples)
            for (int r = 0; r < 4; ++r) {
                if (v > p) mask |= 8u >> r;
                p = v;
                w.put(q + r, v);
                advance();
                v = wc.template of<NX>(x);
                dv |= diverged(v);
            }
        }
        int m = K;
        if (__builtin_expect(dv, 0)) {  // the samples up to the one before the divergent one count
            for (m = 1; m < q && !diverged(w.at(0, m));) ++m;
            mask >>= q - m;
            p = w.at(0, m - 1);
        }
        const unsigned cand = PeakWindow::candidates(mask, up, m);
        const unsigned moved = open != 0u && (mask != 0u || p != w.at(0, -1)) ? 1u : 0u;
        if ((cand | moved) != 0u) w.judge(i, cand, 0u, m, 0, moved, open, on_peak);
        if (dv) break;
        up = mask & 1u;
        w.put(-2, w.at(0, K - 2));
        w.put(-1, p);
    }
    if (!dv) {
        unsigned mask = 0;
        int m = 0;
        for (; i + m < B && !dv;) {
#pragma unroll
            for (int j = 0; j < NX; ++j) xp[j] = x[j];
            mask = (mask << 1) | (v > p ? 1u : 0u);
            p = v;
            w.put(m++, v);
            advance();
            v = wc.template of<NX>(x);
            dv = diverged(v);
        }
        if (m > 0) {
            const unsigned cand = PeakWindow::candidates(mask, up, m);
            if ((cand | open) != 0u) w.judge(i, cand, 0u, m, 0, open, open, on_peak);
        }
    }
    last = p;
    n = w.detector(0).n;
    return dv ? 0 : 1;
}

// The recorded part of a bifurcation point, from its state x after a
// transient that ended bounded and not fixed: nB samples through the
// streaming peak detector (intervals in units hI), divergence and fixed-point
// tests; writes flags/counts/first and the first `cap` kept peaks/intervals
// of row o. FP32 judges windows of samples (record_windows; the steps a
// window runs past a divergent one change nothing that is reported; the
// launch brings Window<1>::bytes of shared memory), FP64 one sample at a time.
template <int S, class T, int W>
__device__ __forceinline__ void bif_record(const SweepParams& P, const BifOut& O, T* x, const T* a,
                                           const StepCtx<T>& c, int nB, double hI, long long o, Component<W> wc) {
    constexpr int NX = Traits<S>::NX;
    T xp[NX];
    int flag = 1;
    int n = 0;  // detected peaks
    const double first = (double)wc.template of<NX>(x);
    double* pk = O.peaks ? O.peaks + o * (long long)O.cap : nullptr;
    double* iv = O.intervals ? O.intervals + o * (long long)O.cap : nullptr;
    auto write_peak = [&](int found, int tprev, T val, int t) {
        if (found >= 1) {
            const int q = found - 1;
            if (q < O.cap) {
                if (pk) pk[q] = (double)val;
                if (iv) iv[q] = __dmul_rn((double)(t - tprev), hI);
            }
        }
    };
#pragma unroll
    for (int j = 0; j < NX; ++j) xp[j] = x[j];
    if constexpr (std::is_same<T, float>::value) {
        float last;
        flag = record_windows<NX, KnownComponent<S, T>::value, Straight<S>::kSamples>(
            nB, x, xp, wc, Window<1>(), last, n, [&] { step<S>(x, a, c); },
            [&](float v) { return bif_diverged(v, P); },
            [&](int, const PeakWindow& d, float val, int t) { write_peak(d.n, d.tprev, val, t); });
    } else {
        PeakStream<T> ps;
        ps.init();
        T v = wc.template of<NX>(x);  // the recorded sample, carried from one step to the next
        for (int i = 0; i < nB; ++i) {
#pragma unroll
            for (int j = 0; j < NX; ++j) xp[j] = x[j];
            T val;
            int t;
            if (ps.push(v, val, t)) {
                write_peak(ps.n, ps.tprev, val, t);
                ps.tprev = t;
                ++ps.n;
            }
            step<S>(x, a, c);
            v = wc.template of<NX>(x);
            if (bif_diverged(v, P)) { flag = 0; break; }
        }
        n = ps.n;
    }
    if (flag == 1 && nB > 0 && bif_fixed<NX>(x, xp)) flag = -1;
    const int kept = n > 1 ? n - 1 : 0;
    O.flags[o] = flag;
    O.counts[o] = flag == 1 ? kept : (flag == -1 ? -1 : 0);
    if (O.first) O.first[o] = first;
}

// ---------------------------------------------------------------------------
// Bifurcation point (reference kernels calculateTransTimeCUDA +
// calculateDiscreteModelCUDA + peakFinderCUDA, bifurcationCUDA.cu:258-371),
// fused. Writes flags/counts/first and the first `cap` kept peaks/intervals.
// Started: all steps of the transient but the last have been run
// (transient_slices.cuh), with the state and flag in start[o].
template <int S, class T, int W, bool Started = false>
__device__ __forceinline__ void bif_point(const SweepParams& P, const BifOut& O, long long p, long long o,
                                             Component<W> wc, const float4* start = nullptr) {
    constexpr int NX = Traits<S>::NX, NA = Traits<S>::NA;
    T x[NX], a[NA], xp[NX];
    load_point<S, T>(P, p, x, a);
    double hp = P.h, hI = P.hInterval;
    int nS = P.S, nB = P.B;
    if (P.sweepStep) {  // this point's own step and step counts, as the host derives them from h
        hp = grid_value(P.grid, p, 0);
        nS = (int)__ddiv_rn(P.transientTime, hp);
        nB = (int)__ddiv_rn(__ddiv_rn(P.tMax, hp), (double)P.bPre);
        hI = __dmul_rn(hp, (double)P.bPre);
    }
    const StepCtx<T> c((T)hp);
    int flag = 1;
    if (nS > 0) {
        // the state before the last step is kept for the fixed-point test:
        // the last step is peeled off the loop, so the others copy nothing
        int s = 0;
        if constexpr (Started) {
            const float4 v = start[o];
            x[0] = v.x;
            x[1] = v.y;
            x[2] = v.z;
            flag = v.w != 0.f ? 1 : 0;
            s = nS - 1;
        } else
        if constexpr (S != SYS_USER) {
            // blocks of kTransientBlock steps, one divergence branch a block:
            // a point's flags do not depend on the step at which it diverged
            // (the steps after it on an unbounded state report nothing).
            // Lorenz in FP32, one warp per scheduler: 69 cycles a step
            // against 91 with a branch after every step.
            constexpr int K = std::is_same<T, float>::value ? Straight<S>::kTransient : kTransientBlock;
            for (; s + K <= nS - 1; s += K) {
                bool dv = false;
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    step<S>(x, a, c);
                    dv |= bif_diverged(wc.template of<NX>(x), P);
                }
                if (dv) { flag = 0; break; }
            }
        }
        if (flag == 1)
            for (; s < nS - 1; ++s) {
                step<S>(x, a, c);
                if (bif_diverged(wc.template of<NX>(x), P)) { flag = 0; break; }
            }
        if (flag == 1) {
#pragma unroll
            for (int j = 0; j < NX; ++j) xp[j] = x[j];
            step<S>(x, a, c);
            if (bif_diverged(wc.template of<NX>(x), P)) flag = 0;
            else if (bif_fixed<NX>(x, xp)) flag = -1;
        }
    }
    if (flag == 1) {
        bif_record<S, T>(P, O, x, a, c, nB, hI, o, wc);
    } else {  // a transient that ended diverged or fixed is reported as diverged
        O.flags[o] = 0;
        O.counts[o] = 0;
        if (O.first) O.first[o] = 0.0;
    }
}

// Bifurcation point of the legacy library's analyses (P.legacyLoop, FP64),
// with the legacy per-point loop in place of the current library's.
// P.legacyLoop 1, the grids over initial conditions or parameters
// (calculateDiscreteModelICCUDA, debri/cudaLibrary.cu:1022-1116, over
// loopCalculateDiscreteModel_int, :604-680, then peakFinderCUDA, :1345-1367):
//  - the transient (one step a sample, no bound) ends the point with flag 0
//    when state component 0 becomes NaN or infinite;
//  - its fixed-point verdict does not stop the recorded part.
// P.legacyLoop 2, the step-size sweep (calculateDiscreteModelCUDA_H,
// :955-1000, over loopCalculateDiscreteModel, :472-527, then
// peakFinderCUDA_H, :1396-1412):
//  - the transient stops early at a NaN or infinite component 0, and its
//    verdict is ignored.
// Both recorded parts take sample x[wv] and then preScaller steps, and test
// the sample for NaN, infinity and |(float)x[wv]| > maxValue (flag 0). The
// change of state over the last sample, s = sum of squared differences,
// marks a fixed point (flag -1, count -1):
//  - loop 1: when sqrt(|s|) < 1e-9;
//  - loop 2: when s == 0 or sqrt(s) < 1e-12 (the legacy keeps no peaks).
// Peaks and intervals (units h * preScaller) are written as in bif_record.
template <int S>
__device__ __forceinline__ void bif_point_legacy(const SweepParams& P, const BifOut& O, long long p, long long o) {
    constexpr int NX = Traits<S>::NX, NA = Traits<S>::NA;
    double x[NX], a[NA], xp[NX];
    load_point<S, double>(P, p, x, a);
    double hp = P.h, hI = P.hInterval;
    int nS = P.S, nB = P.B;
    if (P.sweepStep) {
        hp = grid_value(P.grid, p, 0);
        nS = (int)__ddiv_rn(P.transientTime, hp);
        nB = (int)__ddiv_rn(__ddiv_rn(P.tMax, hp), (double)P.bPre);
        hI = __dmul_rn(hp, (double)P.bPre);
    }
    const StepCtx<double> c(hp);
    const int wv = P.wv, pre = P.bPre;
    auto nan_or_inf = [](double v) {
        return ((unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull) > 0x7fefffffffffffffull;
    };
    int flag = 1;
    for (int s = 0; s < nS; ++s) {
        step<S>(x, a, c);
        if (nan_or_inf(x[0])) {
            if (P.legacyLoop == 1) flag = 0;
            break;
        }
    }
    PeakStream<double> ps;
    ps.init();
    double* pk = O.peaks ? O.peaks + o * (long long)O.cap : nullptr;
    double* iv = O.intervals ? O.intervals + o * (long long)O.cap : nullptr;
    auto on_peak = [&](double val, int t) {
        if (ps.n >= 1) {
            const int q = ps.n - 1;
            if (q < O.cap) {
                if (pk) pk[q] = val;
                if (iv) iv[q] = __dmul_rn((double)(t - ps.tprev), hI);
            }
        }
        ps.tprev = t;
        ++ps.n;
    };
    double first = 0.0;
    if (flag == 1) {
        double v = pick<NX>(x, wv);
        first = v;
        for (int i = 0; i < nB; ++i) {
#pragma unroll
            for (int j = 0; j < NX; ++j) xp[j] = x[j];
            double val;
            int t;
            if (ps.push(v, val, t)) on_peak(val, t);
            for (int r = 0; r < pre; ++r) step<S>(x, a, c);
            v = pick<NX>(x, wv);
            if (basins_diverged(v, P)) { flag = 0; break; }
        }
        if (flag == 1 && nB > 0) {
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < NX; ++j) {
                const double d = __dsub_rn(x[j], xp[j]);
                s = __dadd_rn(s, __dmul_rn(d, d));
            }
            const bool fixed = P.legacyLoop == 1 ? __dsqrt_rn(fabs(s)) < 1e-9 : (s == 0.0 || __dsqrt_rn(s) < 1e-12);
            if (fixed) flag = -1;
        }
    }
    const int kept = ps.n > 1 ? ps.n - 1 : 0;
    O.flags[o] = flag;
    O.counts[o] = flag == 1 ? kept : (flag == -1 ? -1 : 0);
    if (O.first) O.first[o] = flag == -1 ? first : 0.0;
}

// Sums over the kept peaks of a basins point: peak values and intervals.
// FP64 path: the reference's per-peak FP64 sums (avgPeakFinderCUDA,
// basinsCUDA.cu:818-864). FP32 path: no FP64 instruction per peak (the FP64
// pipe of this GPU is a small fraction of the FP32 rate): the values are
// summed as an unevaluated float pair with the error-free TwoSum (about 48
// significant bits), the intervals as the integer time span they telescope
// to, and both are widened to FP64 once at the end.
template <class T> struct PeakSums;
template <> struct PeakSums<double> {
    double sp = 0.0, si = 0.0;
    __device__ __forceinline__ void add(double val, int dt, double hI) {
        sp = sp + val;
        si = si + __dmul_rn((double)dt, hI);
    }
    __device__ __forceinline__ double peaks() const { return sp; }
    __device__ __forceinline__ double intervals(double) const { return si; }
};
template <> struct PeakSums<float> {
    float hi = 0.f, lo = 0.f;
    int span = 0;
    __device__ __forceinline__ void add(float val, int dt) {
        const float s = hi + val;  // TwoSum(hi, val) = s + err exactly
        const float bv = s - hi;
        const float err = (hi - (s - bv)) + (val - bv);
        hi = s;
        lo = lo + err;
        span += dt;
    }
    __device__ __forceinline__ void store(float4* to) const { *to = make_float4(hi, lo, __int_as_float(span), 0.f); }
    __device__ __forceinline__ void load(const float4* from) {
        const float4 v = *from;
        hi = v.x;
        lo = v.y;
        span = __float_as_int(v.z);
    }
    static __device__ __forceinline__ void add_stored(float4* at, float val, int dt) {
        PeakSums s;
        s.load(at);
        s.add(val, dt);
        s.store(at);
    }
    __device__ __forceinline__ double peaks() const { return (double)hi + (double)lo; }
    __device__ __forceinline__ double intervals(double hI) const { return __dmul_rn((double)span, hI); }
};

// The results of a basins point: kept peaks, the sums of their values and
// intervals, the last recorded sample. Called by every lane of the warp that
// has a point to write (they fold the clustering's keys together).
__device__ __forceinline__ void write_basins_point(const BasinsOut& O, long long o, int flag, int kept, double peaks,
                                                   double intervals, double last) {
    double ap, ai;
    if (flag == 0) { ap = 999.0; ai = 999.0; }
    else if (flag == -1) { ap = last; ai = -1.0; }
    else if (kept <= 0) { ap = 1000.0; ai = 1000.0; }
    else { ap = peaks / (double)kept; ai = intervals / (double)kept; }
    O.flags[o] = flag;
    O.avgPeaks[o] = ap;
    O.avgIntervals[o] = ai;
    if (O.counts) O.counts[o] = flag == 1 ? kept : 0;
    if (O.last) O.last[o] = last;
    if (O.mm) {  // the clustering's normalisation bounds
        FeatureKeys fk;
        fk.add(flag, flag == 1 ? kept : 0, ap, ai, last);
        fk.flush(O.mm);
    }
}

// ---------------------------------------------------------------------------
// Basins point (reference calculateTransTimeCUDA + calculateDiscreteModelCUDA
// + avgPeakFinderCUDA, basinsCUDA.cu:233-314 and 818-864), fused. PRE1: the
// sweep has preScaller == 1 (one step per sample, no inner loop).
// The recorded part of a basins point, from its state x after the transient:
// peak detector, divergence and fixed-point tests, features into row o.
template <int S, class T, bool PRE1, int W>
__device__ __forceinline__ void basins_record(const SweepParams& P, const BasinsOut& O, T* x, const T* a,
                                              const StepCtx<T>& c, long long o, Component<W> wc) {
    constexpr int NX = Traits<S>::NX;
    T xp[NX];
#pragma unroll
    for (int j = 0; j < NX; ++j) xp[j] = x[j];
    int flag = 1, n = 0;  // n: detected peaks
    PeakSums<T> sums;
    T lastT = T(0);  // widened once after the loop (a per-step FP64 convert costs FP64-pipe time)
    auto advance = [&] {
        if (PRE1) step<S>(x, a, c);
        else
            for (int r = 0; r < P.preScaller; ++r) step<S>(x, a, c);
    };
    if constexpr (std::is_same<T, float>::value) {  // as bif_record; the sums in shared memory
        const Window<1> w;
        sums.store(w.sum);
        constexpr bool stop = !(KnownComponent<S, T>::value && PRE1);
        constexpr int samples = PRE1 ? Straight<S>::kSamples : Straight<S>::kLongSamples;
        flag = record_windows<NX, stop, samples>(
            P.B, x, xp, wc, w, lastT, n, advance, [&](float v) { return basins_diverged(v, P); },
            [&](int, const PeakWindow& d, float val, int t) {
                if (d.n >= 1) PeakSums<float>::add_stored(w.sum, val, t - d.tprev);
            });
        sums.load(w.sum);
    } else {
        PeakStream<T> ps;
        ps.init();
        T v = wc.template of<NX>(x);  // the recorded sample, carried from one step to the next
        for (int i = 0; i < P.B; ++i) {
#pragma unroll
            for (int j = 0; j < NX; ++j) xp[j] = x[j];
            lastT = v;
            T val;
            int t;
            if (ps.push(v, val, t)) {
                if (ps.n >= 1) sums.add(val, t - ps.tprev, P.hInterval);
                ps.tprev = t;
                ++ps.n;
            }
            advance();
            v = wc.template of<NX>(x);
            if (basins_diverged(v, P)) { flag = 0; break; }
        }
        n = ps.n;
    }
    if (flag == 1 && P.B > 0 && basins_fixed<NX>(x, xp)) flag = -1;
    write_basins_point(O, o, flag, n > 1 ? n - 1 : 0, sums.peaks(), sums.intervals(P.hInterval), (double)lastT);
}

template <int S, class T, bool PRE1, int W, bool Started = false>
__device__ __forceinline__ void basins_point(const SweepParams& P, const BasinsOut& O, long long p, long long o,
                                             Component<W> wc, const float4* start = nullptr) {
    constexpr int NX = Traits<S>::NX, NA = Traits<S>::NA;
    T x[NX], a[NA];
    load_point<S, T>(P, p, x, a);
    const StepCtx<T> c((T)P.h);
    if constexpr (Started) {  // the transient has been run (transient_slices.cuh)
        const float4 v = start[o];
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
    } else {
        for (int s = 0; s < P.S; ++s) step<S>(x, a, c);
    }
    basins_record<S, T, PRE1>(P, O, x, a, c, o, wc);
}

// ---------------------------------------------------------------------------
// LLE point, the reference's Benettin scheme (LLECUDA.cu:114-166) in full
// precision T for both trajectories: calcBlocks+1 blocks of NT steps of x and
// of its twin q; d = |x-q|/eps; sum += log(d); q = x - (x-q)/d; sum / tMax.
// The twin starts at x + eps along state component 0.
// State and parameters of point p of an LLE-type sweep: a 1-D grid (p = i)
// or the 2-D map (p = j*nPts + i), over parameters values[mut] or initial
// conditions ic[mut] (L.mutateState); the second dimension is written last.
// Swept values are linspace start + n*step, multiply and add rounded apart.
template <int NX, int NA, class T>
__device__ __forceinline__ void lle_load(const LleParams& L, long long p, T* x, T* a) {
    const long long i = L.dim == 1 ? p : p % L.nPts, j = L.dim == 1 ? 0 : p / L.nPts;
    const double va = L.table[0]    ? L.table[0][i]
                      : L.nPts == 1 ? L.rangeA[0]
                                    : __dadd_rn(L.rangeA[0], __dmul_rn((double)i, L.stepA));
    const double vb = L.table[1]                      ? L.table[1][j]
                      : (L.nPts == 1 || L.dim == 1) ? L.rangeB[0]
                                                    : __dadd_rn(L.rangeB[0], __dmul_rn((double)j, L.stepB));
#pragma unroll
    for (int k = 0; k < NX; ++k) {
        double v = L.ic[k];
        if (L.mutateState) {
            if (k == L.mut[0]) v = va;
            if (k == L.mut[1]) v = vb;
        }
        x[k] = (T)v;
    }
#pragma unroll
    for (int k = 0; k < NA; ++k) {
        double v = L.values[k];
        if (!L.mutateState) {
            if (k == L.mut[0]) v = va;
            if (k == L.mut[1]) v = vb;
        }
        a[k] = (T)v;
    }
}

// The Benettin blocks of the reference's calculateSystem (LLE/src/LLECUDA.cu:
// 146-162) from an orbit x and a full twin trajectory q: calcBlocks + 1
// blocks of ntp steps of each, dist = sqrt(sum (x - q)^2) / eps, sum +=
// log(dist), q = x - (x - q) / dist; the sum over tMax.
template <int S, class T>
__device__ __forceinline__ double lle_benettin_full(const LleParams& L, T* x, T* q, const T* a) {
    constexpr int NX = Traits<S>::NX;
    const StepCtx<T> c((T)L.h);
    double sum = 0.0;
    for (int b = 0; b <= L.calcBlocks; ++b) {
        for (int s = 0; s < L.ntp; ++s) step<S>(x, a, c);
        for (int s = 0; s < L.ntp; ++s) step<S>(q, a, c);
        double dist = 0.0;
#pragma unroll
        for (int k = 0; k < NX; ++k) {
            const double df = (double)x[k] - (double)q[k];
            dist = dist + df * df;
        }
        dist = sqrt(dist) / L.eps;
        sum = sum + log(dist);
#pragma unroll
        for (int k = 0; k < NX; ++k) q[k] = (T)((double)x[k] - (((double)x[k] - (double)q[k]) / dist));
    }
    return sum / L.tMax;
}

template <int S, class T>
__device__ __forceinline__ double lle_point_full(const LleParams& L, long long p) {
    constexpr int NX = Traits<S>::NX, NA = Traits<S>::NA;
    T x[NX], q[NX], a[NA];
    lle_load<NX, NA>(L, p, x, a);
    const StepCtx<T> c((T)L.h);
    for (int s = 0; s < L.trans; ++s) step<S>(x, a, c);
#pragma unroll
    for (int k = 0; k < NX; ++k) q[k] = x[k];
    if (L.twin == 1) {
        // the reference's twin start (LLECUDA.cu:97-101): a float FMA of a unit
        // direction times eps onto the float-rounded state, here with the
        // direction e_x instead of its cuRAND draw
#pragma unroll
        for (int k = 0; k < NX; ++k) q[k] = (T)__fmaf_rn(k == 0 ? 1.0f : 0.0f, (float)L.eps, (float)x[k]);
    } else {
        q[0] = x[0] + (T)L.eps;
    }
    return lle_benettin_full<S>(L, x, q, a);
}

// LLE point with the twin carried as the exact difference e = q - x (only for
// the quadratic RK4 systems): x and e in FP32 registers. Same block count and
// division by tMax as above. How the stretch of every block is measured and
// the twin renormalised is the Stretch mode:
//   kRenormPow2 (default): e is scaled by a power of two 2^-k that brings |e|
//     back to within a factor sqrt(2) of eps -- exact in FP32 -- and k is
//     summed as an integer, so the sum of the blocks' log-stretches telescopes
//     exactly to k ln 2 + log(|e_final| / eps), taken once in FP64 from the
//     FP64 norm of the final e (ff.h);
//   kRenormF32Log: log2(|e|^2 / eps^2) per block on the SFU (__log2f), e
//     rescaled to length eps with rsqrtf, the logs summed in FP32 over groups
//     of kLleGroup blocks and the group sums in FP64;
//   kRenormF64: the reference's arithmetic (LLE/src/LLECUDA.cu:146-162):
//     dist = sqrt(sum (x - p)^2) / eps in FP64, sum += log(dist), e /= dist.
enum LleRenorm { kRenormPow2 = 0, kRenormF32Log = 1, kRenormF64 = 2 };
constexpr int kLleGroup = 16;

__device__ __forceinline__ double nan_if_not_finite(double v) {
    return isfinite(v) ? v : __longlong_as_double(0x7ff8000000000000LL);
}

template <int RN> struct Stretch;
template <> struct Stretch<kRenormPow2> {
    double eps;  // the stretch of every block is measured against eps, as the reference measures it
    int eps2Exp, k = 0;
    double v = 0.0;
    __device__ __forceinline__ explicit Stretch(double eps_) : eps(eps_) {
        const float e0 = (float)eps_;
        eps2Exp = (int)((__float_as_uint(e0 * e0) >> 23) & 0xff) - 126;
    }
    __device__ __forceinline__ float renorm(float e0_, float e1, float e2) {
        const int j = pow2_rescale_exponent(fmaf(e0_, e0_, fmaf(e1, e1, e2 * e2)), eps2Exp);
        k += j;
        return pow2_scale(j);
    }
    __device__ __forceinline__ void last(float e0_, float e1, float e2) {
        const double n2 = (double)e0_ * e0_ + (double)e1 * e1 + (double)e2 * e2;
        v = pow2_log_stretch(k, n2, eps);
    }
    __device__ __forceinline__ double result(double tMax) const { return nan_if_not_finite(v / tMax); }
};
template <> struct Stretch<kRenormF32Log> {
    float eps, inv_eps2, part = 0.f;
    int cnt = 0;
    double sum = 0.0;  // sum of log2(d^2)
    __device__ __forceinline__ Stretch(float eps_, double epsd) : eps(eps_), inv_eps2((float)(1.0 / (epsd * epsd))) {}
    __device__ __forceinline__ float add(float n2) {
        part += __log2f(n2 * inv_eps2);
        if (++cnt == kLleGroup) {
            sum += (double)part;
            part = 0.f;
            cnt = 0;
        }
        return n2;
    }
    __device__ __forceinline__ float renorm(float e0, float e1, float e2) {
        const float n2 = add(fmaf(e0, e0, fmaf(e1, e1, e2 * e2)));
        return eps * rsqrtf(n2);
    }
    __device__ __forceinline__ void last(float e0, float e1, float e2) { add(fmaf(e0, e0, fmaf(e1, e1, e2 * e2))); }
    __device__ __forceinline__ double result(double tMax) const {
        return (sum + (double)part) * (0.5 * 0.69314718055994530942) / tMax;  // log2(d^2) -> ln(d)
    }
};
template <> struct Stretch<kRenormF64> {
    double eps, sum = 0.0;
    __device__ __forceinline__ explicit Stretch(double eps_) : eps(eps_) {}
    __device__ __forceinline__ double dist(float e0, float e1, float e2) const {
        return sqrt((double)e0 * e0 + (double)e1 * e1 + (double)e2 * e2) / eps;
    }
    __device__ __forceinline__ float renorm(float e0, float e1, float e2) {
        const double d = dist(e0, e1, e2);
        sum += log(d);
        return (float)(1.0 / d);
    }
    __device__ __forceinline__ void last(float e0, float e1, float e2) { sum += log(dist(e0, e1, e2)); }
    __device__ __forceinline__ double result(double tMax) const { return sum / tMax; }
};
template <int RN> __device__ __forceinline__ Stretch<RN> make_stretch(const LleParams& L);
template <> __device__ __forceinline__ Stretch<kRenormPow2> make_stretch<kRenormPow2>(const LleParams& L) {
    return Stretch<kRenormPow2>(L.eps);
}
template <> __device__ __forceinline__ Stretch<kRenormF32Log> make_stretch<kRenormF32Log>(const LleParams& L) {
    return Stretch<kRenormF32Log>((float)L.eps, L.eps);
}
template <> __device__ __forceinline__ Stretch<kRenormF64> make_stretch<kRenormF64>(const LleParams& L) {
    return Stretch<kRenormF64>(L.eps);
}

template <class F, class T>
__device__ __forceinline__ void twin_steps(T* x, T* e, const T* a, const RK4H<T>& c, int n) {  // n steps, 2 per trip
    int s = 0;
    for (; s + 2 <= n; s += 2) {
        rk4_step_twin<F>(x, e, a, c);
        rk4_step_twin<F>(x, e, a, c);
    }
    if (s < n) rk4_step_twin<F>(x, e, a, c);
}

// The Benettin blocks b0 to b1 - 1 of an FP32 twin carried as a difference e
// (three state components): steps(e, n) advances the orbit and e by n steps.
template <int RN, class Steps>
__device__ __forceinline__ void lle_twin_blocks(const LleParams& L, float* e, Stretch<RN>& st, int b0, int b1,
                                                Steps&& steps) {
    const int nb = L.calcBlocks + 1;
    for (int b = b0; b < b1; ++b) {
        steps(e, L.ntp);
        if (b + 1 < nb) {
            const float r = st.renorm(e[0], e[1], e[2]);
            e[0] *= r;
            e[1] *= r;
            e[2] *= r;
        } else {
            st.last(e[0], e[1], e[2]);
        }
    }
}

// A map's point (or pair of points) as its kernels run it: from its start
// through the transient and the blocks to its result, in one go or a slice of
// the horizon at a time (lle_slices.h), between which words() hands its state
// to io.
template <class Point>
__device__ __forceinline__ void run_point(const LleParams& L, long long p, long long q, double* outp, double* outq) {
    Point z(L, p, q);
    z.transient(L.trans);
    z.blocks(L, 0, L.calcBlocks + 1);
    z.result(L, outp, outq);
}

// FP32 LLE point of an RK4 system.
template <class F> struct LlePoint {
    static constexpr int kPoints = 1, kWords = 7;
    float x[3], e[3], a[3];
    const RK4H<float> c;
    Stretch<kRenormPow2> st;
    __device__ __forceinline__ LlePoint(const LleParams& L, long long p, long long)
        : c((float)L.h), st(make_stretch<kRenormPow2>(L)) {
        lle_load<3, 3>(L, p, x, a);
        e[0] = (float)L.eps;
        e[1] = 0.f;
        e[2] = 0.f;
    }
    __device__ __forceinline__ void transient(int n) {
        for (int s = 0; s < n; ++s) rk4_step<F>(x, a, c);
    }
    __device__ __forceinline__ void blocks(const LleParams& L, int b0, int b1) {
        lle_twin_blocks(L, e, st, b0, b1, [&](float* d, int n) { twin_steps<F>(x, d, a, c, n); });
    }
    template <class IO> __device__ __forceinline__ void words(IO& io) {
        io.word(x);
        io.word(e);
        io.word(st.k);
    }
    __device__ __forceinline__ void result(const LleParams& L, double* outp, double*) const {
        *outp = st.result(L.tMax);
    }
};
template <class F>
__device__ __forceinline__ double lle_point_twin(const LleParams& L, long long p) {
    double v;
    run_point<LlePoint<F>>(L, p, p, &v, nullptr);
    return v;
}

// The FP32 LLE point of Chameleon (the reference's default system): the twin
// as the difference of chameleon_step_twin.
__device__ __forceinline__ double lle_point_twin_chameleon(const LleParams& L, long long p) {
    float x[3], a[7];
    lle_load<3, 7>(L, p, x, a);
    const float h = (float)L.h;
    for (int s = 0; s < L.trans; ++s) chameleon_step<float>(x, a, h);
    float e[3] = {(float)L.eps, 0.f, 0.f};
    auto st = make_stretch<kRenormPow2>(L);
    lle_twin_blocks(L, e, st, 0, L.calcBlocks + 1, [&](float* d, int n) {
        for (int s = 0; s < n; ++s) chameleon_step_twin<float>(x, d, a, h);
    });
    return st.result(L.tMax);
}

// ---------------------------------------------------------------------------
// Lyapunov spectrum of one point: one twin per state dimension, started along
// the unit vectors (x + eps e_j), integrated NT at a time beside the base
// trajectory; after every block the differences y_j - x are orthogonalised by
// classical Gram-Schmidt (b_j = d_j - sum_{m<j} (d_j.b_m / b_m.b_m) b_m), each
// norm |b_j| adds log(|b_j| / eps) to exponent j and the twins restart at
// x + eps b_j/|b_j| -- the scheme of the legacy library's spectrum kernel
// (debri/cudaLibrary.cu:2141-2330). Blocks and the division by tMax are the
// LLE map's (calcBlocks + 1 blocks), so exponent 0 estimates the same
// quantity as lle_point_full. out[p*NX + j] = exponent j.
template <int S>
__device__ __forceinline__ void spectrum_point_full(const LleParams& L, long long p, double* out) {
    constexpr int N = Traits<S>::NX, NA = Traits<S>::NA;
    double x[N], y[N][N], a[NA], sum[N];
    lle_load<N, NA>(L, p, x, a);
    const StepCtx<double> c(L.h);
    for (int s = 0; s < L.trans; ++s) step<S>(x, a, c);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        sum[j] = 0.0;
#pragma unroll
        for (int i = 0; i < N; ++i) y[j][i] = i == j ? x[i] + L.eps : x[i];
    }
    for (int b = 0; b <= L.calcBlocks; ++b) {
        for (int s = 0; s < L.ntp; ++s) step<S>(x, a, c);
#pragma unroll
        for (int j = 0; j < N; ++j)
            for (int s = 0; s < L.ntp; ++s) step<S>(y[j], a, c);
        double d[N][N], g[N][N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                d[j][i] = y[j][i] - x[i];
                g[j][i] = d[j][i];
            }
#pragma unroll
            for (int m = 0; m < j; ++m) {
                double num = 0.0, den = 0.0;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    num = num + d[j][i] * g[m][i];
                    den = den + g[m][i] * g[m][i];
                }
                const double frac = den == 0.0 ? 0.0 : num / den;
#pragma unroll
                for (int i = 0; i < N; ++i) g[j][i] = g[j][i] - frac * g[m][i];
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double n2 = 0.0;
#pragma unroll
            for (int i = 0; i < N; ++i) n2 = n2 + g[j][i] * g[j][i];
            const double nrm = sqrt(n2);
            sum[j] = sum[j] + log(nrm / L.eps);
#pragma unroll
            for (int i = 0; i < N; ++i) y[j][i] = x[i] + (nrm == 0.0 ? 0.0 : g[j][i] / nrm) * L.eps;
        }
    }
#pragma unroll
    for (int j = 0; j < N; ++j) out[p * N + j] = sum[j] / L.tMax;
}

// The spectrum in FP32 for the quadratic RK4 systems and Chameleon: the twins
// carried as exact differences e_j, Gram-Schmidt in FP32, per block
// log2(|b_j|^2/eps^2) on the SFU summed in FP32 groups of kLleGroup blocks and
// added into FP64, as the FP32 LLE map does. steps(e, n) advances the orbit
// and the three differences by n steps.
__device__ __forceinline__ void spectrum_start(const LleParams& L, float (*e)[3], double* sum) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int i = 0; i < 3; ++i) e[j][i] = i == j ? (float)L.eps : 0.f;
        sum[j] = 0.0;
    }
}
__device__ __forceinline__ double spectrum_result(const LleParams& L, double sum) {
    return sum * (0.5 * 0.69314718055994530942) / L.tMax;
}
// Blocks from to to - 1; from is a multiple of kLleGroup.
template <class Steps>
__device__ __forceinline__ void spectrum_twin_blocks(const LleParams& L, float (*e)[3], double* sum, int from, int to,
                                                     Steps&& steps) {
    const float eps = (float)L.eps;
    const float inv_eps2 = (float)(1.0 / (L.eps * L.eps));
    for (int b0 = from; b0 < to; b0 += kLleGroup) {
        const int bn = min(kLleGroup, to - b0);
        float part[3] = {0.f, 0.f, 0.f};
        for (int b = 0; b < bn; ++b) {
            steps(e, L.ntp);
            float g[3][3];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
#pragma unroll
                for (int i = 0; i < 3; ++i) g[j][i] = e[j][i];
#pragma unroll
                for (int m = 0; m < j; ++m) {
                    const float num = fmaf(e[j][0], g[m][0], fmaf(e[j][1], g[m][1], e[j][2] * g[m][2]));
                    const float den = fmaf(g[m][0], g[m][0], fmaf(g[m][1], g[m][1], g[m][2] * g[m][2]));
                    const float frac = den == 0.f ? 0.f : num / den;
#pragma unroll
                    for (int i = 0; i < 3; ++i) g[j][i] = fmaf(-frac, g[m][i], g[j][i]);
                }
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float n2 = fmaf(g[j][0], g[j][0], fmaf(g[j][1], g[j][1], g[j][2] * g[j][2]));
                part[j] += __log2f(n2 * inv_eps2);
                const float r = n2 > 0.f ? eps * rsqrtf(n2) : 0.f;
#pragma unroll
                for (int i = 0; i < 3; ++i) e[j][i] = g[j][i] * r;
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) sum[j] += (double)part[j];
    }
}

// Results three to a point, at outp.
template <class F> struct SpectrumPoint {
    static constexpr int kPoints = 1, kWords = 18;
    float x[3], a[3], e[3][3];
    double sum[3];
    const RK4H<float> c;
    __device__ __forceinline__ SpectrumPoint(const LleParams& L, long long p, long long) : c((float)L.h) {
        lle_load<3, 3>(L, p, x, a);
        spectrum_start(L, e, sum);
    }
    __device__ __forceinline__ void transient(int n) {
        for (int s = 0; s < n; ++s) rk4_step<F>(x, a, c);
    }
    __device__ __forceinline__ void blocks(const LleParams& L, int b0, int b1) {
        spectrum_twin_blocks(L, e, sum, b0, b1, [&](float (*d)[3], int n) {
            for (int s = 0; s < n; ++s) rk4_step_multi<F, 3>(x, d, a, c);
        });
    }
    template <class IO> __device__ __forceinline__ void words(IO& io) {
        io.word(x);
        io.word(e);
        io.word(sum);
    }
    __device__ __forceinline__ void result(const LleParams& L, double* outp, double*) const {
#pragma unroll
        for (int j = 0; j < 3; ++j) outp[j] = spectrum_result(L, sum[j]);
    }
};

__device__ __forceinline__ void spectrum_point_twin_chameleon(const LleParams& L, long long p, double* out) {
    float x[3], a[7];
    lle_load<3, 7>(L, p, x, a);
    const float h = (float)L.h;
    for (int s = 0; s < L.trans; ++s) chameleon_step<float>(x, a, h);
    float e[3][3];
    double sum[3];
    spectrum_start(L, e, sum);
    spectrum_twin_blocks(L, e, sum, 0, L.calcBlocks + 1, [&](float (*d)[3], int n) {
        for (int s = 0; s < n; ++s) chameleon_step_multi<float, 3>(x, d, a, h);
    });
#pragma unroll
    for (int j = 0; j < 3; ++j) out[p * 3 + j] = spectrum_result(L, sum[j]);
}

// ---------------------------------------------------------------------------
// Packed pair of FP32 values: two trajectories advanced by one instruction
// stream with Blackwell's paired FP32 instructions (fma.rn.f32x2,
// add.rn.f32x2, mul.rn.f32x2). Each lane of the pair is rounded exactly as
// the scalar FP32 operation would be; the pair halves the instructions the
// schedulers issue for the same flops.
struct P2 {
    float2 v;
    __device__ __forceinline__ P2() {}
    __device__ __forceinline__ explicit P2(double s) : v(make_float2((float)s, (float)s)) {}
    __device__ __forceinline__ P2(float a, float b) : v(make_float2(a, b)) {}
};
__device__ __forceinline__ P2 mk(float2 f) { P2 r; r.v = f; return r; }
__device__ __forceinline__ P2 operator+(P2 a, P2 b) { return mk(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ P2 operator-(P2 a) { return mk(make_float2(-a.v.x, -a.v.y)); }
__device__ __forceinline__ P2 operator-(P2 a, P2 b) { return mk(__fadd2_rn(a.v, make_float2(-b.v.x, -b.v.y))); }
__device__ __forceinline__ P2 operator*(P2 a, P2 b) { return mk(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ P2& operator*=(P2& a, P2 b) { a = a * b; return a; }
__device__ __forceinline__ P2 fmaT(P2 a, P2 b, P2 c) { return mk(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ P2 addR(P2 a, P2 b) { return a + b; }
// Word operations of float-float pairs of packed lanes (ff.h): each one
// paired instruction, rounded per lane exactly as the scalar operation;
// a - b as fma(b, -1, a), which is RN(a - b) in one instruction.
__device__ __forceinline__ P2 w_add(P2 a, P2 b) { return mk(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ P2 w_sub(P2 a, P2 b) { return mk(__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)); }
__device__ __forceinline__ P2 w_mul(P2 a, P2 b) { return mk(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ P2 w_fma(P2 a, P2 b, P2 c) { return mk(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ P2 w_neg(P2 a) { return mk(make_float2(-a.v.x, -a.v.y)); }

// Step constants of a packed pair: rounded exactly as RK4H<float> rounds them.
template <> struct RK4H<P2> {
    P2 h, hh, h6;
    __device__ __forceinline__ explicit RK4H(float h_)
        : h((double)h_), hh((double)(h_ * 0.5f)), h6((double)(h_ / 6.0f)) {}
};

// Two LLE points per thread (indices p and q), lanes of P2. Same arithmetic
// per lane as LlePoint; the per-block stretch and renormalisation (Stretch
// mode RN) run per lane.
template <class F, int RN = kRenormPow2> struct LlePair {
    static constexpr int kPoints = 2, kWords = 14;
    P2 x[3], e[3], a[3];
    const RK4H<P2> c;
    Stretch<RN> s0, s1;
    __device__ __forceinline__ LlePair(const LleParams& L, long long p, long long q)
        : c((float)L.h), s0(make_stretch<RN>(L)), s1(make_stretch<RN>(L)) {
        float xs[2][3], as[2][3];
        lle_load<3, 3>(L, p, xs[0], as[0]);
        lle_load<3, 3>(L, q, xs[1], as[1]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a[k] = P2(as[0][k], as[1][k]);
            x[k] = P2(xs[0][k], xs[1][k]);
        }
        const float eps = (float)L.eps;
        e[0] = P2((double)eps);
        e[1] = P2(0.0);
        e[2] = P2(0.0);
    }
    __device__ __forceinline__ void transient(int n) {
        for (int s = 0; s < n; ++s) rk4_step<F>(x, a, c);
    }
    __device__ __forceinline__ void blocks(const LleParams& L, int b0, int b1) {
        const int nb = L.calcBlocks + 1;
        for (int b = b0; b < b1; ++b) {
            twin_steps<F>(x, e, a, c, L.ntp);
            if (b + 1 < nb) {
                const P2 r(s0.renorm(e[0].v.x, e[1].v.x, e[2].v.x), s1.renorm(e[0].v.y, e[1].v.y, e[2].v.y));
                e[0] *= r;
                e[1] *= r;
                e[2] *= r;
            } else {
                s0.last(e[0].v.x, e[1].v.x, e[2].v.x);
                s1.last(e[0].v.y, e[1].v.y, e[2].v.y);
            }
        }
    }
    template <class IO> __device__ __forceinline__ void words(IO& io) {
        io.word(x);
        io.word(e);
        io.word(s0.k);
        io.word(s1.k);
    }
    __device__ __forceinline__ void result(const LleParams& L, double* outp, double* outq) const {
        *outp = s0.result(L.tMax);
        if (outq) *outq = s1.result(L.tMax);
    }
};

// Two spectrum points per thread (indices p and q), lanes of P2: SpectrumPoint
// per lane, Gram-Schmidt packed too, with the
// divisions, logs and reciprocal roots per lane.
template <class F> struct SpectrumPair {
    static constexpr int kPoints = 2, kWords = 36;
    P2 x[3], a[3], e[3][3];
    double sum[2][3];
    const RK4H<P2> c;
    __device__ __forceinline__ SpectrumPair(const LleParams& L, long long p, long long q) : c((float)L.h) {
        float xs[2][3], as[2][3];
        lle_load<3, 3>(L, p, xs[0], as[0]);
        lle_load<3, 3>(L, q, xs[1], as[1]);
        const float eps = (float)L.eps;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a[k] = P2(as[0][k], as[1][k]);
            x[k] = P2(xs[0][k], xs[1][k]);
            sum[0][k] = sum[1][k] = 0.0;
#pragma unroll
            for (int i = 0; i < 3; ++i) e[k][i] = i == k ? P2(eps, eps) : P2(0.0);
        }
    }
    __device__ __forceinline__ void transient(int n) {
        for (int s = 0; s < n; ++s) rk4_step<F>(x, a, c);
    }
    template <class IO> __device__ __forceinline__ void words(IO& io) {
        io.word(x);
        io.word(e);
        io.word(sum);
    }
    __device__ __forceinline__ void result(const LleParams& L, double* outp, double* outq) const {
#pragma unroll
        for (int j = 0; j < 3; ++j) outp[j] = spectrum_result(L, sum[0][j]);
        if (outq) {
#pragma unroll
            for (int j = 0; j < 3; ++j) outq[j] = spectrum_result(L, sum[1][j]);
        }
    }
    __device__ __forceinline__ void blocks(const LleParams& L, int from, int to);
};
template <class F> __device__ __forceinline__ void SpectrumPair<F>::blocks(const LleParams& L, int from, int to) {
    const float eps = (float)L.eps;
    const float inv_eps2 = (float)(1.0 / (L.eps * L.eps));
    for (int b0 = from; b0 < to; b0 += kLleGroup) {
        const int bn = min(kLleGroup, to - b0);
        P2 part[3] = {P2(0.0), P2(0.0), P2(0.0)};
        for (int b = 0; b < bn; ++b) {
            for (int s = 0; s < L.ntp; ++s) rk4_step_multi<F, 3>(x, e, a, c);
#pragma unroll
            for (int j = 1; j < 3; ++j) {
                // e[m] for m < j hold the orthogonal vectors already; the
                // projections take the vector as it was before them
                const P2 d[3] = {e[j][0], e[j][1], e[j][2]};
#pragma unroll
                for (int m = 0; m < j; ++m) {
                    const P2* g = e[m];
                    const P2 num = fmaT(d[0], g[0], fmaT(d[1], g[1], d[2] * g[2]));
                    const P2 den = fmaT(g[0], g[0], fmaT(g[1], g[1], g[2] * g[2]));
                    const P2 frac(den.v.x == 0.f ? -0.f : -(num.v.x / den.v.x),
                                  den.v.y == 0.f ? -0.f : -(num.v.y / den.v.y));
#pragma unroll
                    for (int i = 0; i < 3; ++i) e[j][i] = fmaT(frac, g[i], e[j][i]);
                }
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const P2 n2 = fmaT(e[j][0], e[j][0], fmaT(e[j][1], e[j][1], e[j][2] * e[j][2]));
                part[j] = part[j] + P2(__log2f(n2.v.x * inv_eps2), __log2f(n2.v.y * inv_eps2));
                const P2 r(n2.v.x > 0.f ? eps * rsqrtf(n2.v.x) : 0.f, n2.v.y > 0.f ? eps * rsqrtf(n2.v.y) : 0.f);
#pragma unroll
                for (int i = 0; i < 3; ++i) e[j][i] *= r;
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            sum[0][j] += (double)part[j].v.x;
            sum[1][j] += (double)part[j].v.y;
        }
    }
}

// ---------------------------------------------------------------------------
// Two bifurcation / basins points per thread in packed FP32x2 lanes (RK4
// systems). Each lane keeps its own flag, peak detector and outputs and
// follows exactly the scalar FP32 path: a lane that diverges stops recording
// while the pair keeps stepping (its state is then ignored), and the loop
// ends when neither lane is recording.
__device__ __forceinline__ float lane(const P2& v, int l) { return l ? v.v.y : v.v.x; }

// sqrtf(fabsf(sum (x - xp)^2)) < 1e-9 per lane, as bif_fixed<NX, float>
template <int NX> __device__ __forceinline__ bool bif_fixed_lane(const P2* x, const P2* xp, int l) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NX; ++j) {
        const float d = lane(x[j], l) - lane(xp[j], l);
        s = s + d * d;
    }
    return (double)sqrtf(fabsf(s)) < 1e-9;
}
template <int NX> __device__ __forceinline__ bool basins_fixed_lane(const P2* x, const P2* xp, int l) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NX; ++j) {
        const float d = lane(x[j], l) - lane(xp[j], l);
        s = s + d * d;
    }
    return sqrt(fabs((double)s)) < 1e-9;
}

template <class F>
__device__ __forceinline__ void load_pair(const SweepParams& P, long long p0, long long p1, P2* x, P2* a) {
    float xs[2][3], as[2][3];
    load_point<SYS_LORENZ_RK4, float>(P, p0, xs[0], as[0]);  // any 3-state, 3-parameter system loads alike
    load_point<SYS_LORENZ_RK4, float>(P, p1, xs[1], as[1]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        x[k] = P2(xs[0][k], xs[1][k]);
        a[k] = P2(as[0][k], as[1][k]);
    }
}

// The transient of two bifurcation points in packed FP32x2 lanes, the last
// step peeled off for the fixed-point test; flag[l] (1 on entry for a lane in
// use, 0 otherwise) ends 1, 0 (diverged) or -1 (fixed), as bif_point's.
// Blocks of kTransientBlock steps with one test a block, as in bif_point.
template <class F, int W>
__device__ __forceinline__ void bif_pair_transient(const SweepParams& P, P2* x, const P2* a, int* flag,
                                                   Component<W> wc) {
    P2 xp[3];
    if (P.S > 0) {
        const RK4H<P2> c((float)P.h);
        int s = 0;
        {  // blocks of kTransientBlock steps with one test a block, as in bif_point
            constexpr int K = kTransientBlock;
            for (; s + K <= P.S - 1; s += K) {
                bool d0 = false, d1 = false;
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    rk4_step<F>(x, a, c);
                    const P2 v = wc.template of<3>(x);
                    d0 |= bif_diverged(v.v.x, P);
                    d1 |= bif_diverged(v.v.y, P);
                }
                if (d0) flag[0] = 0;
                if (d1) flag[1] = 0;
                if (flag[0] != 1 && flag[1] != 1) break;
            }
        }
        if (flag[0] == 1 || flag[1] == 1)
            for (; s < P.S - 1; ++s) {  // the last step peeled off, as in bif_point
                rk4_step<F>(x, a, c);
                const P2 v = wc.template of<3>(x);
                if (flag[0] == 1 && bif_diverged(v.v.x, P)) flag[0] = 0;
                if (flag[1] == 1 && bif_diverged(v.v.y, P)) flag[1] = 0;
                if (flag[0] != 1 && flag[1] != 1) break;
            }
        if (flag[0] == 1 || flag[1] == 1) {
#pragma unroll
            for (int j = 0; j < 3; ++j) xp[j] = x[j];
            rk4_step<F>(x, a, c);
            const P2 v = wc.template of<3>(x);
            if (flag[0] == 1 && bif_diverged(v.v.x, P)) flag[0] = 0;
            if (flag[1] == 1 && bif_diverged(v.v.y, P)) flag[1] = 0;
#pragma unroll
            for (int l = 0; l < 2; ++l)
                if (flag[l] == 1 && bif_fixed_lane<3>(x, xp, l)) flag[l] = -1;
        }
    }
}

// The recorded loop of two trajectories in packed lanes, per lane exactly
// record_windows: rec[l] says whether lane l records, flag[l] becomes 0 when
// it diverges (the pair goes on while the other lane records), xp the state
// before the last advance (of a lane that did not diverge).
// Tested: the first four samples are tested one by one. A basins transient has
// no test, and where it left both orbits of a pair beyond the bound a window
// run past the first sample would be most of the pair's time: 700^2 Lorenz
// points, all of them beyond, 5 steps a sample, 0.116 -> 0.042 ms. (A test after
// every four samples of a window costs the other maps 2 %; the bifurcation's
// pairs, whose transient has a test, lose up to 5 % to this form.)
template <bool Tested, int W, class Advance, class Diverged, class OnPeak>
__device__ __forceinline__ void record_pair_windows(int B, P2* x, P2* xp, Component<W> wc, const Window<2>& w, bool* rec,
                                                    int* flag, float* last, Advance&& advance, Diverged&& diverged,
                                                    OnPeak&& on_peak) {
    constexpr int K = Window<2>::K;
    PeakWindow d;
    d.init();
    w.keep(0, d);
    w.keep(1, d);
    w.put(-2, make_float2(0.f, 0.f));
    w.put(-1, make_float2(0.f, 0.f));
    P2 v = wc.template of<3>(x), p(0.0);
    unsigned up0 = 0, up1 = 0, open = 0;
    int i = 0;
    auto carry = [&](unsigned mask0, unsigned mask1, int n) {
        // a lane that diverged on a plateau leaves it there: nothing of it is judged any more
        open &= (rec[0] ? 1u : 0u) | (rec[1] ? 2u : 0u);
        up0 = mask0 & 1u;
        up1 = mask1 & 1u;
        w.put(-2, make_float2(w.at(0, n - 2), w.at(1, n - 2)));
        w.put(-1, p.v);
    };
    // full windows, their steps without a test; whether a lane still records
    auto windows = [&]() -> bool {
        for (; i + K < B; i += K) {
            unsigned mask0 = 0, mask1 = 0;
            bool dv0 = false, dv1 = false;
#pragma unroll 1
            for (int q = 0; q < K; q += 4) {
                mask0 <<= 4;
                mask1 <<= 4;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    if (v.v.x > p.v.x) mask0 |= 8u >> r;
                    if (v.v.y > p.v.y) mask1 |= 8u >> r;
                    p = v;
                    w.put(q + r, v.v);
                    advance();
                    v = wc.template of<3>(x);
                    dv0 |= diverged(v.v.x);
                    dv1 |= diverged(v.v.y);
                }
            }
            int m0 = K, m1 = K;
            if (__builtin_expect(rec[0] && dv0, 0)) {
                for (m0 = 1; m0 < K && !diverged(w.at(0, m0));) ++m0;
                mask0 >>= K - m0;
            }
            if (__builtin_expect(rec[1] && dv1, 0)) {
                for (m1 = 1; m1 < K && !diverged(w.at(1, m1));) ++m1;
                mask1 >>= K - m1;
            }
            const unsigned c0 = rec[0] ? PeakWindow::candidates(mask0, up0, m0) : 0u;
            const unsigned c1 = rec[1] ? PeakWindow::candidates(mask1, up1, m1) : 0u;
            unsigned moved = 0;
            if (open != 0u)
                moved = open & ((mask0 != 0u || w.at(0, m0 - 1) != w.at(0, -1) ? 1u : 0u) |
                                (mask1 != 0u || w.at(1, m1 - 1) != w.at(1, -1) ? 2u : 0u));
            if ((c0 | c1 | moved) != 0u) w.judge(i, c0, c1, m0, m1, moved, open, on_peak);
            if (rec[0]) last[0] = w.at(0, m0 - 1);
            if (rec[1]) last[1] = w.at(1, m1 - 1);
            if (rec[0] && dv0) {
                rec[0] = false;
                flag[0] = 0;
            }
            if (rec[1] && dv1) {
                rec[1] = false;
                flag[1] = 0;
            }
            if (!rec[0] && !rec[1]) return false;
            carry(mask0, mask1, K);
        }
        return true;
    };
    // a window of at most `most` samples, a test after each; whether samples and a lane that records are left
    auto tested = [&](int most) -> bool {
        unsigned mask0 = 0, mask1 = 0;
        int m0 = 0, m1 = 0, m = 0;  // samples each lane judges, and those of the window
        for (; m < most && i + m < B && (rec[0] || rec[1]);) {
#pragma unroll
            for (int j = 0; j < 3; ++j) xp[j] = x[j];
            if (rec[0]) {
                mask0 = (mask0 << 1) | (v.v.x > p.v.x ? 1u : 0u);
                ++m0;
                last[0] = v.v.x;
            }
            if (rec[1]) {
                mask1 = (mask1 << 1) | (v.v.y > p.v.y ? 1u : 0u);
                ++m1;
                last[1] = v.v.y;
            }
            p = v;
            w.put(m++, v.v);
            advance();
            v = wc.template of<3>(x);
            if (rec[0] && diverged(v.v.x)) { rec[0] = false; flag[0] = 0; }
            if (rec[1] && diverged(v.v.y)) { rec[1] = false; flag[1] = 0; }
        }
        const unsigned c0 = m0 > 0 ? PeakWindow::candidates(mask0, up0, m0) : 0u;
        const unsigned c1 = m1 > 0 ? PeakWindow::candidates(mask1, up1, m1) : 0u;
        if ((c0 | c1 | open) != 0u) w.judge(i, c0, c1, m0, m1, open, open, on_peak);
        i += m;
        if (i >= B || (!rec[0] && !rec[1])) return false;
        carry(mask0, mask1, m);
        return true;
    };
    if constexpr (Tested) {
        for (int most = 4; tested(most) && windows(); most = K) {}
    } else if (windows()) {
        tested(K);
    }
}

template <class F, int W>
__device__ __forceinline__ void bif_pair_point(const SweepParams& P, const BifOut& O, long long p0, long long p1,
                                                  long long o0, long long o1, bool two, Component<W> wc) {
    P2 x[3], a[3], xp[3];
    load_pair<F>(P, p0, p1, x, a);
    const RK4H<P2> c((float)P.h);
    int flag[2] = {1, two ? 1 : 0};
    bif_pair_transient<F>(P, x, a, flag, wc);
    bool rec[2];
    double first[2] = {0.0, 0.0};  // stays 0 for a lane that does not record (as the scalar path)
    int n[2] = {0, 0};  // detected peaks
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        rec[l] = flag[l] == 1;
        if (!rec[l]) flag[l] = 0;
    }
    const long long oo[2] = {o0, o1};
    if (rec[0] || rec[1]) {
        {
            const P2 v = wc.template of<3>(x);
            if (rec[0]) first[0] = (double)v.v.x;
            if (rec[1]) first[1] = (double)v.v.y;
        }
        const Window<2> w;
        float last[2];
        record_pair_windows<false>(P.B, x, xp, wc, w, rec, flag, last, [&] { rk4_step<F>(x, a, c); },
                            [&](float v) { return bif_diverged(v, P); },
                            [&](int l, const PeakWindow& d, float val, int t) {
                                const int q = d.n - 1;
                                if (q >= 0 && q < O.cap) {
                                    const long long at = (l ? o1 : o0) * O.cap + q;
                                    if (O.peaks) O.peaks[at] = (double)val;
                                    if (O.intervals) O.intervals[at] = __dmul_rn((double)(t - d.tprev), P.hInterval);
                                }
                            });
        n[0] = w.detector(0).n;
        n[1] = w.detector(1).n;
#pragma unroll
        for (int l = 0; l < 2; ++l)
            if (rec[l] && P.B > 0 && bif_fixed_lane<3>(x, xp, l)) flag[l] = -1;
    }
#pragma unroll
    for (int l = 0; l < (two ? 2 : 1); ++l) {
        const int kept = n[l] > 1 ? n[l] - 1 : 0;
        O.flags[oo[l]] = flag[l];
        O.counts[oo[l]] = flag[l] == 1 ? kept : (flag[l] == -1 ? -1 : 0);
        if (O.first) O.first[oo[l]] = first[l];
    }
}

template <class F, bool PRE1, int W>
__device__ __forceinline__ void basins_pair_point(const SweepParams& P, const BasinsOut& O, long long p0,
                                                     long long p1, long long o0, long long o1, bool two,
                                                     Component<W> wc) {
    P2 x[3], a[3], xp[3];
    load_pair<F>(P, p0, p1, x, a);
    const RK4H<P2> c((float)P.h);
    for (int s = 0; s < P.S; ++s) rk4_step<F>(x, a, c);
#pragma unroll
    for (int j = 0; j < 3; ++j) xp[j] = x[j];
    int flag[2] = {1, two ? 1 : 0};
    bool rec[2] = {true, two};
    PeakSums<float> sums[2];
    float lastF[2] = {0.f, 0.f};  // widened after the loop
    const Window<2> w;
    sums[0].store(w.sum);
    sums[1].store(w.sum + blockDim.x);
    record_pair_windows<true>(
        P.B, x, xp, wc, w, rec, flag, lastF,
        [&] {
            if (PRE1) rk4_step<F>(x, a, c);
            else
                for (int r = 0; r < P.preScaller; ++r) rk4_step<F>(x, a, c);
        },
        [&](float v) { return basins_diverged(v, P); },
        [&](int l, const PeakWindow& d, float val, int t) {
            if (d.n >= 1) PeakSums<float>::add_stored(w.sum + l * blockDim.x, val, t - d.tprev);
        });
    const int n[2] = {w.detector(0).n, w.detector(1).n};
    sums[0].load(w.sum);
    sums[1].load(w.sum + blockDim.x);
    const long long oo[2] = {o0, o1};
    FeatureKeys fk;
#pragma unroll
    for (int l = 0; l < (two ? 2 : 1); ++l) {
        if (rec[l] && P.B > 0 && basins_fixed_lane<3>(x, xp, l)) flag[l] = -1;
        const double last = (double)lastF[l];
        const int kept = n[l] > 1 ? n[l] - 1 : 0;
        double ap, ai;
        if (flag[l] == 0) { ap = 999.0; ai = 999.0; }
        else if (flag[l] == -1) { ap = last; ai = -1.0; }
        else if (kept <= 0) { ap = 1000.0; ai = 1000.0; }
        else { ap = sums[l].peaks() / (double)kept; ai = sums[l].intervals(P.hInterval) / (double)kept; }
        O.flags[oo[l]] = flag[l];
        O.avgPeaks[oo[l]] = ap;
        O.avgIntervals[oo[l]] = ai;
        if (O.counts) O.counts[oo[l]] = flag[l] == 1 ? kept : 0;
        if (O.last) O.last[oo[l]] = last;
        fk.add(flag[l], flag[l] == 1 ? kept : 0, ap, ai, last);
    }
    if (O.mm) fk.flush(O.mm);
}

// ---------------------------------------------------------------------------
// Trajectory recorder: nSteps steps of one trajectory per thread, writing the
// state before the first step and after every step.
template <int S, class T>
__device__ __forceinline__ void trajectory_point(const double* x0, const double* a0, double h, int nSteps,
                                                 double* out, long long t) {
    constexpr int NX = Traits<S>::NX, NA = Traits<S>::NA;
    T x[NX], a[NA];
#pragma unroll
    for (int j = 0; j < NX; ++j) x[j] = (T)x0[t * NX + j];
#pragma unroll
    for (int j = 0; j < NA; ++j) a[j] = (T)a0[t * NA + j];
    const StepCtx<T> c((T)h);
    double* o = out + t * (long long)(nSteps + 1) * NX;
#pragma unroll
    for (int j = 0; j < NX; ++j) o[j] = (double)x[j];
    auto record = [&](int s) {
        step<S>(x, a, c);
#pragma unroll
        for (int j = 0; j < NX; ++j) o[(long long)s * NX + j] = (double)x[j];
    };
    if constexpr (std::is_same<T, float>::value && S <= SYS_CHEN_RK4) {
        // one step at a time: several in a row are scheduled for a longer chain (64
        // trajectories, 4,000 steps: Lorenz 0.73 -> 0.64 ms, Rossler 0.69 -> 0.63, Chen
        // 0.72 -> 0.63)
#pragma unroll 1
        for (int s = 1; s <= nSteps; ++s) record(s);
    } else {
        for (int s = 1; s <= nSteps; ++s) record(s);
    }
}

}  // namespace chaos
