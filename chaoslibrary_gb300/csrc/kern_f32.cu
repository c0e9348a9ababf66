// FP32 kernels: trajectories in FP32 registers (contraction allowed), peak
// times, intervals and means in FP64. The LLE kernel carries the twin as the
// exact difference e = q - x (quadratic RK4 systems only) and accumulates the
// log-stretch sum in FP64.
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "engine.cuh"
#include "lle_slices.h"
#include "transient_slices.cuh"
#include "sweep_launch.h"

namespace chaos {

namespace {
constexpr int kBlock = kSweepBlock;

// The sweep kernels take Window<trajectories per thread>::bytes(block)
// of dynamic shared memory.
template <int S, int W, bool Started = false>
__global__ void __launch_bounds__(kMaxBlock) bif_kernel_f32(SweepParams P, BifOut O, const float4* start) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= P.nPoints) return;
    bif_point<S, float, W, Started>(P, O, P.pBegin + o, o, Component<W>{P.wv}, start);
}

template <int S>
__global__ void __launch_bounds__(kBlock) bif_list_kernel_f32(SweepParams P, BifOut O, const int* list, int count) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    bif_point<S, float>(P, O, list[k], k, Component<-1>{P.wv});
}

// MINB = resident blocks per SM the register allocation is shaped for:
// 12 (40 registers, 48 warps/SM) or 16 (32 registers, 64 warps/SM, a few
// bytes of spill outside the step loop). Picked per system by the tuner.
template <class F, int MINB>
__global__ void __launch_bounds__(kBlock, MINB) lle_twin_kernel_f32(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    out[o] = lle_point_twin<F>(L, L.pBegin + o);
}

__global__ void __launch_bounds__(kBlock) spectrum_chameleon_kernel_f32(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    spectrum_point_twin_chameleon(L, L.pBegin + o, out);
}

__global__ void __launch_bounds__(kBlock) lle_chameleon_kernel_f32(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    out[o] = lle_point_twin_chameleon(L, L.pBegin + o);
}

template <int S>
__global__ void __launch_bounds__(kBlock) trajectory_kernel_f32(const double* x0, const double* a0, double h, int nSteps,
                                                       double* out, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    trajectory_point<S, float>(x0, a0, h, nSteps, out, t);
}

// Two points per thread in packed FP32x2 lanes, the first `singles` blocks one.
// Bound by the FMA pipe; 124 registers (Lorenz), four blocks per SM. 7.58 rows of
// Lorenz points per SM, 3,510 steps: 3.31 ms asked for three blocks, 3.35 asked
// for none or four, 3.89 at six (80 registers: spills).
template <class F>
__global__ void __launch_bounds__(kBlock, 3) spectrum_pair_kernel_f32(LleParams L, double* out, unsigned singles) {
    bool pair;
    const long long o = mixed_point(singles, pair);
    if (o >= L.nPoints) return;
    const long long p = L.pBegin + o;
    const bool two = pair && o + 1 < L.nPoints;
    double* outp = out + 3 * p;
    if (pair) run_point<SpectrumPair<F>>(L, p, two ? p + 1 : p, outp, two ? outp + 3 : nullptr);
    else run_point<SpectrumPoint<F>>(L, p, p, outp, nullptr);
}

// Bifurcation / basins, two points per thread in packed FP32x2 lanes (RK4
// systems). Bound by the FMA pipe. Registers capped at 80: six blocks of 128
// per SM, as many as the sample windows leave room for.
template <class F, int W>
__global__ void __launch_bounds__(kMaxBlock, 3) bif_pair_kernel_f32(SweepParams P, BifOut O) {
    const long long o = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
    if (o >= P.nPoints) return;
    const bool two = o + 1 < P.nPoints;
    bif_pair_point<F>(P, O, P.pBegin + o, P.pBegin + (two ? o + 1 : o), o, two ? o + 1 : o, two, Component<W>{P.wv});
}

inline unsigned grid_for(long long n) { return (unsigned)((n + kBlock - 1) / kBlock); }
}  // namespace
namespace {

// Variant of the FP32 LLE kernel: 12 / 16 = one point per thread shaped for
// 12 or 16 resident blocks per SM; 2 = two points per thread in packed
// FP32x2 lanes. CHAOS_LLE_MINB forces one; otherwise the pair kernel runs, with
// the blocks that single_blocks says on one point per thread.
std::atomic<int> g_lle_variant{0};

int lle_env_variant() {
    static int forced = [] {
        const char* s = getenv("CHAOS_LLE_MINB");
        return s ? atoi(s) : 0;
    }();
    return forced;
}

// 0: none is forced
int lle_forced_variant() {
    const int set = g_lle_variant.load(std::memory_order_relaxed);
    return set ? set : lle_env_variant();
}

}  // namespace

std::atomic<int> g_sweep_pairs{-1};

// Paired (two points per thread, packed FP32x2 lanes) FP32 sweeps for the RK4
// systems. Mode 1 (default): sweeps of at least 2048 points per SM run as
// pairs, smaller ones one point per thread: pairs issue half the instructions
// but halve the warps that hide each other's latency, and up to those 16 rows
// of 128 the transient of single points runs in slices. Measured on GB300, one
// point per thread against pairs: 1-D Rossler, 20,000 steps, 160,000 points
// 4.97 / 5.16 ms, 240,000 7.24 / 7.10, 320,000 9.41 / 9.06, 700,001 19.7 / 17.8;
// Lorenz basins, 25,000 steps, 400^2 5.73 / 5.95 ms, 500^2 8.48 / 8.23, 600^2
// 12.3 / 11.7, 1024^2 34.6 / 31.2 (so full maps of 1,400 to 2,048 points per SM
// would be up to 10 % faster in pairs). 2 (or 3): always pairs; 0: never. Set
// with chaos_set_tuning or CHAOS_SWEEP_PAIRS.
int sweep_pairs() {
    const int v = g_sweep_pairs.load(std::memory_order_relaxed);
    if (v >= 0) return v;
    static int env = [] {
        const char* s = getenv("CHAOS_SWEEP_PAIRS");
        const int m = s ? atoi(s) : 1;
        return m < 0 || m > 3 ? 1 : m;
    }();
    return env;
}
int set_sweep_pairs(int v) {
    if (v < 0 || v > 3) return -1;
    g_sweep_pairs.store(v);
    return 0;
}

// Launch shapes the self-timing tuner (tune.cu) found, per kind (0 1-D
// bifurcation, 1 basins, 2 LLE map) and RK4 system: 0 = none (the built-in
// rules below), else form * 1024 + block with form 1 (one point per thread)
// or 2 (two points per thread in packed FP32x2 lanes); for the LLE map also form
// 12 / 16 (one point per thread, registers shaped for 12 / 16 resident blocks per
// SM, block 128).
std::atomic<int> g_shape[3][3];

int shape_of(int kind, int system) {
    return system >= 0 && system <= SYS_CHEN_RK4 ? g_shape[kind][system].load(std::memory_order_relaxed) : 0;
}

long long pair_threshold() { return 2048 * sm_count(); }

// Pairs halve the threads: worth it when the sweep fills the GPU several
// times over, not for small (latency-bound) sweeps. An explicit sweep-pairs
// mode (0 / 2) wins; then a tuned shape; then the measured rule.
Launch sweep_launch(const SweepParams& P, bool basins) {
    if (P.system > SYS_CHEN_RK4 || P.sweepStep) return {1, kBlock};  // a pair shares one step size
    const int mode = sweep_pairs();
    const int shape = shape_of(basins ? 1 : 0, P.system);
    const int block = shape ? shape % 1024 : kBlock;
    const bool big = P.nPoints >= pair_threshold();
    if (mode == 0) return {1, block};
    if (mode >= 2) return {2, block};
    if (!big) return {1, kBlock};  // (the tuner times 8192 points per SM)
    return {shape ? shape / 1024 : 2, block};
}

template <class F> void launch_bif_pairs(const SweepParams& P, const BifOut& O, int block, cudaStream_t st) {
    with_component<true>(P.wv, [&](auto wc) {
        auto* k = bif_pair_kernel_f32<F, decltype(wc)::kIndex>;
        const size_t shm = Window<2>::bytes(block);
        if (shm > 48 * 1024)  // blocks of 256 (the tuner's)
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
        k<<<grid_of((P.nPoints + 1) / 2, block), block, shm, st>>>(P, O);
    });
    note_launch();
}

template <int S, int W>
void launch_bif_points_as(const SweepParams& P, const BifOut& O, int block, float4* state, cudaStream_t st) {
    auto* k = bif_kernel_f32<S, W>;
    if constexpr (KnownComponent<S, float>::value) {
        const TransientPlan plan = state ? transient_plan(P, false) : TransientPlan{};
        if (plan.jobs > 0) {
            launch_transient<S, W, false>(plan, P, state, st);
            k = bif_kernel_f32<S, W, true>;
        }
    }
    k<<<grid_of(P.nPoints, block), block, Window<1>::bytes(block), st>>>(P, O, state);
    note_launch();
}
template <int S>
void launch_bif_points(const SweepParams& P, const BifOut& O, int block, float4* state, cudaStream_t st) {
    with_component<KnownComponent<S, float>::value>(
        P.wv, [&](auto wc) { launch_bif_points_as<S, decltype(wc)::kIndex>(P, O, block, state, st); });
}

size_t transient_state_bytes(const SweepParams& P, bool basins) { return transient_plan(P, basins).bytes(); }

cudaError_t launch_bif_f32(const SweepParams& P, const BifOut& O, cudaStream_t st, float4* state) {
    if (P.nPoints <= 0) return cudaSuccess;
    const Launch l = sweep_launch(P, false);
    if (l.form == 2) {
        if (P.system == SYS_LORENZ_RK4) launch_bif_pairs<Lorenz>(P, O, l.block, st);
        else if (P.system == SYS_ROSSLER_RK4) launch_bif_pairs<Rossler>(P, O, l.block, st);
        else launch_bif_pairs<Chen>(P, O, l.block, st);
        return cudaGetLastError();
    }
#define CALL(S) launch_bif_points<S>(P, O, l.block, state, st)
    CHAOS_SYSTEM_SWITCH(P.system, CALL)
#undef CALL
    return cudaGetLastError();
}

cudaError_t launch_bif_list_f32(const SweepParams& P, const BifOut& O, const int* list, int count, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
#define CALL(S) \
    (bif_list_kernel_f32<S><<<grid_for(count), kBlock, Window<1>::bytes(kBlock), st>>>(P, O, list, count), note_launch())
    CHAOS_SYSTEM_SWITCH(P.system, CALL)
#undef CALL
    return cudaGetLastError();
}

// Two points per thread in packed FP32x2 lanes. Registers capped at 56 (three
// resident blocks of 384 threads): nine blocks of 128 per SM instead of eight
// at the 62 the kernel takes unbounded. The cap costs a few bytes of spills
// outside the step loop; the 1024^2 Rössler map went from 133.7 to 128.6 ms
// (from 3.37 waves of resident blocks to 2.99) and the Lorenz map from 39.1
// to 36.2 ms, results unchanged. Blocks of 64, 128 and 256 (the tuner's
// choices) all launch under the bound.
// Mixed: the first `singles` blocks run one point per thread (single_blocks).
// Chen's step keeps more than Lorenz's and Rossler's: its mixed form takes 80
// registers (three rows of 128 points per SM, 5,510 steps, 1.14 ms at 56, 1.11 at
// 80), and where it has more than two rows and no singles it runs in a form of
// pairs alone at 56 (mixed / pairs alone: 2 rows 0.741 / 0.747 ms, 4 rows 1.40 /
// 1.37, 30 rows 9.99 / 9.60; the others' mixed form runs pairs as fast as one of
// pairs alone, or faster).
template <class F> constexpr bool is_chen() { return std::is_same<F, Chen>::value; }
template <class F, int RN = kRenormPow2, bool Mixed = RN == kRenormPow2>
__global__ void __launch_bounds__(is_chen<F>() && Mixed ? kMaxBlock : 384, is_chen<F>() && Mixed ? 2 : 3)
lle_pair_kernel_f32(LleParams L, double* out, unsigned singles) {
    bool pair;
    const long long o = mixed_point(singles, pair);
    if (o >= L.nPoints) return;
    if (Mixed && !pair) {
        out[o] = lle_point_twin<F>(L, L.pBegin + o);
        return;
    }
    const bool two = o + 1 < L.nPoints;
    run_point<LlePair<F, RN>>(L, L.pBegin + o, L.pBegin + (two ? o + 1 : o), out + o, two ? out + o + 1 : nullptr);
}

// A slice of the jobs whose turn it is (lle_slices.h). At the 56 registers of
// the kernel above this one spills in its loops, and a launch never has more
// than four blocks per SM: 4.2 rows of Lorenz points, 10,510 steps, 2.99 ms at
// 56 registers, 2.91 at 80, 2.85 at 128 (unsliced 3.06). The spectrum likewise:
// 8.2 rows, 3,510 steps, 3.73 ms at 128 registers, 3.65 above (unsliced 4.14).
template <class F>
__global__ void __launch_bounds__(kBlock, 4) lle_slice_kernel_f32(LleParams L, SlicePlan plan, long long turn,
                                                                  float* state, double* out) {
    run_slice<LlePair<F>, LlePoint<F>>(L, plan, turn, state, out, 1);
}
template <class F>
__global__ void __launch_bounds__(kBlock, 2) spectrum_slice_kernel_f32(LleParams L, SlicePlan plan, long long turn,
                                                                    float* state, double* out) {
    run_slice<SpectrumPair<F>, SpectrumPoint<F>>(L, plan, turn, state, out + 3 * L.pBegin, 3);
}

// Stretch mode of the FP32 LLE maps of the RK4 systems (LleRenorm): 0 the
// exact power-of-two renormalisation (default); 1 and 2 run the pair kernel
// with the per-block FP32 log or the per-block FP64 norm and log instead.
std::atomic<int> g_lle_renorm{0};

template <class F>
static void launch_twin(const LleParams& L, double* out, cudaStream_t st, int minb, int block, float* state) {
    const int rn = g_lle_renorm.load(std::memory_order_relaxed);
    if (minb == 0 && rn == kRenormPow2 && state) {
        const SlicePlan plan = slice_plan(L, kSliceLle);
        if (plan.jobs > 0) return launch_slices(plan, lle_slice_kernel_f32<F>, L, out, state, st);
    }
    const unsigned gp = grid_of((L.nPoints + 1) / 2, minb == 2 ? block : kBlock);
    const int bp = minb == 2 ? block : kBlock;
    const unsigned singles = single_blocks(L.nPoints);
    const bool mixed = minb == 0 && (!is_chen<F>() || singles || L.nPoints <= 2 * kBlock * sm_count());
    if (rn == kRenormF32Log) lle_pair_kernel_f32<F, kRenormF32Log><<<gp, bp, 0, st>>>(L, out, 0u);
    else if (rn == kRenormF64) lle_pair_kernel_f32<F, kRenormF64><<<gp, bp, 0, st>>>(L, out, 0u);
    else if (mixed) lle_pair_kernel_f32<F><<<mixed_grid(L.nPoints, singles), kBlock, 0, st>>>(L, out, singles);
    else if (minb == 0 || minb == 2) lle_pair_kernel_f32<F, kRenormPow2, !is_chen<F>()><<<gp, bp, 0, st>>>(L, out, 0u);
    else if (minb >= 16) lle_twin_kernel_f32<F, 16><<<grid_for(L.nPoints), kBlock, 0, st>>>(L, out);
    else lle_twin_kernel_f32<F, 12><<<grid_for(L.nPoints), kBlock, 0, st>>>(L, out);
    note_launch();
}

int set_launch_shape(int kind, int system, int code) {
    if (kind < 0 || kind > 2 || system < 0 || system > SYS_CHEN_RK4 || code < 0) return -1;
    g_shape[kind][system].store(code);
    return 0;
}
int get_launch_shape(int kind, int system) {
    return kind >= 0 && kind <= 2 ? shape_of(kind, system) : 0;
}

int set_lle_variant(int v) {
    if (v != 0 && v != 2 && v != 12 && v != 16) return -1;
    g_lle_variant.store(v);
    return 0;
}
int get_lle_variant() { return lle_forced_variant(); }

int set_lle_renorm(int v) {
    if (v < kRenormPow2 || v > kRenormF64) return -1;
    g_lle_renorm.store(v);
    return 0;
}
int get_lle_renorm() { return g_lle_renorm.load(); }

// an explicit variant (chaos_set_tuning / CHAOS_LLE_MINB) wins, then a tuned
// shape, for maps of more rows than those that run in slices or in mixed blocks:
// the tuner times 64 rows per SM; 0: neither
static int lle_form(const LleParams& L, int& block) {
    block = kBlock;
    if (const int forced = lle_forced_variant()) return forced;
    if (L.nPoints <= kSliceLle.mostRows() * kBlock * sm_count()) return 0;
    const int shape = shape_of(2, L.system);
    if (shape / 1024 == 2) block = shape % 1024;
    return shape / 1024;
}

size_t lle_f32_state_bytes(const LleParams& L) {
    int block;
    if (!system_has_difference_form(L.system) || lle_form(L, block) != 0 || get_lle_renorm() != kRenormPow2)
        return 0;
    const SlicePlan plan = slice_plan(L, kSliceLle);
    return plan.words(plan.points == 2 ? LlePair<Lorenz>::kWords : LlePoint<Lorenz>::kWords) * sizeof(float);
}

cudaError_t launch_lle_f32(const LleParams& L, double* out, cudaStream_t st, float* state) {
    if (L.nPoints <= 0) return cudaSuccess;
    int block;
    const int minb = lle_form(L, block);
    switch (L.system) {
        case SYS_LORENZ_RK4: launch_twin<Lorenz>(L, out, st, minb, block, state); break;
        case SYS_ROSSLER_RK4: launch_twin<Rossler>(L, out, st, minb, block, state); break;
        case SYS_CHEN_RK4: launch_twin<Chen>(L, out, st, minb, block, state); break;
        case SYS_CHAMELEON:
            lle_chameleon_kernel_f32<<<grid_for(L.nPoints), kBlock, 0, st>>>(L, out);
            note_launch();
            break;
        default: return cudaErrorNotSupported;
    }
    return cudaGetLastError();
}

template <class F> static void launch_spectrum(const LleParams& L, double* out, cudaStream_t st, float* state) {
    const SlicePlan plan = state ? slice_plan(L, kSliceSpectrum) : SlicePlan{};
    if (plan.jobs > 0) return launch_slices(plan, spectrum_slice_kernel_f32<F>, L, out, state, st);
    // up to three rows all of them single: their time goes with the rows, 2 rows of
    // Lorenz points (2,510 steps) 0.626 ms, in pairs 0.647, 3 rows 0.914, one single
    // and one of pairs 0.935 (Rossler 0.495 / 0.523 and 0.719 / 0.744)
    const unsigned singles = L.nPoints <= kSliceSpectrum.singleRows * kBlock * sm_count()
                                 ? grid_of(L.nPoints, kBlock) : single_blocks(L.nPoints);
    spectrum_pair_kernel_f32<F><<<mixed_grid(L.nPoints, singles), kBlock, 0, st>>>(L, out, singles);
    note_launch();
}

size_t spectrum_f32_state_bytes(const LleParams& L) {
    if (!system_has_difference_form(L.system)) return 0;
    const SlicePlan plan = slice_plan(L, kSliceSpectrum);
    return plan.words(plan.points == 2 ? SpectrumPair<Lorenz>::kWords : SpectrumPoint<Lorenz>::kWords) * sizeof(float);
}

cudaError_t launch_spectrum_f32(const LleParams& L, double* out, cudaStream_t st, float* state) {
    if (L.nPoints <= 0) return cudaSuccess;
    switch (L.system) {
        case SYS_LORENZ_RK4: launch_spectrum<Lorenz>(L, out, st, state); break;
        case SYS_ROSSLER_RK4: launch_spectrum<Rossler>(L, out, st, state); break;
        case SYS_CHEN_RK4: launch_spectrum<Chen>(L, out, st, state); break;
        case SYS_CHAMELEON:
            spectrum_chameleon_kernel_f32<<<grid_for(L.nPoints), kBlock, 0, st>>>(L, out);
            note_launch();
            break;
        default: return cudaErrorNotSupported;
    }
    return cudaGetLastError();
}

cudaError_t launch_trajectory_f32(int system, const double* x0, const double* a0, double h, int nSteps,
                                  double* out, long long n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
#define CALL(S) \
    (trajectory_kernel_f32<S><<<grid_for(n), kBlock, 0, st>>>(x0, a0, h, nSteps, out, n), note_launch())
    CHAOS_SYSTEM_SWITCH(system, CALL)
#undef CALL
    return cudaGetLastError();
}

}  // namespace chaos
