// FP32 basins kernels (FP32 trajectories, peak times, intervals and means in
// FP64): a translation unit of its own so that it compiles beside the other
// FP32 kernels.
#include "engine.cuh"
#include "sweep_launch.h"
#include "transient_slices.cuh"

namespace chaos {

namespace {
// The sweep kernels take Window<trajectories per thread>::bytes(block) of
// dynamic shared memory.
template <int S, bool PRE1, int W, bool Started = false>
__global__ void __launch_bounds__(kMaxBlock) basins_kernel_f32(SweepParams P, BasinsOut O, const float4* start) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= P.nPoints) return;
    basins_point<S, float, PRE1, W, Started>(P, O, P.pBegin + o, o, Component<W>{P.wv}, start);
}

// Two points per thread in packed FP32x2 lanes (RK4 systems); registers capped
// as in the bifurcation's pair kernel.
template <class F, bool PRE1, int W>
__global__ void __launch_bounds__(kMaxBlock, 3) basins_pair_kernel_f32(SweepParams P, BasinsOut O) {
    const long long o = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
    if (o >= P.nPoints) return;
    const bool two = o + 1 < P.nPoints;
    basins_pair_point<F, PRE1>(P, O, P.pBegin + o, P.pBegin + (two ? o + 1 : o), o, two ? o + 1 : o, two,
                               Component<W>{P.wv});
}

// (with preScaller > 1 a sample costs several steps, and picking its component
// at run time is lost in them)
template <class F, bool PRE1>
void launch_basins_pairs_as(const SweepParams& P, const BasinsOut& O, int block, cudaStream_t st) {
    with_component<PRE1>(P.wv, [&](auto wc) {
        auto* k = basins_pair_kernel_f32<F, PRE1, decltype(wc)::kIndex>;
        const size_t shm = Window<2>::bytes(block);
        if (shm > 48 * 1024)  // blocks of 256 (the tuner's)
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
        k<<<grid_of((P.nPoints + 1) / 2, block), block, shm, st>>>(P, O);
    });
    note_launch();
}

template <class F> void launch_basins_pairs(const SweepParams& P, const BasinsOut& O, int block, cudaStream_t st) {
    if (P.preScaller == 1) launch_basins_pairs_as<F, true>(P, O, block, st);
    else launch_basins_pairs_as<F, false>(P, O, block, st);
}

template <int S, bool PRE1, int W>
void launch_basins_points_as(const SweepParams& P, const BasinsOut& O, int block, float4* state, cudaStream_t st) {
    auto* k = basins_kernel_f32<S, PRE1, W>;
    if constexpr (KnownComponent<S, float>::value) {
        const TransientPlan plan = state ? transient_plan(P, true) : TransientPlan{};
        if (plan.jobs > 0) {
            launch_transient<S, -1, true>(plan, P, state, st);
            k = basins_kernel_f32<S, PRE1, W, true>;
        }
    }
    k<<<grid_of(P.nPoints, block), block, Window<1>::bytes(block), st>>>(P, O, state);
    note_launch();
}
template <int S, bool PRE1>
void launch_basins_points(const SweepParams& P, const BasinsOut& O, int block, float4* state, cudaStream_t st) {
    with_component<KnownComponent<S, float>::value && PRE1>(
        P.wv, [&](auto wc) { launch_basins_points_as<S, PRE1, decltype(wc)::kIndex>(P, O, block, state, st); });
}
}  // namespace

cudaError_t launch_basins_f32(const SweepParams& P, const BasinsOut& O, cudaStream_t st, float4* state) {
    if (P.nPoints <= 0) return cudaSuccess;
    const Launch l = sweep_launch(P, true);
    if (l.form == 2) {
        if (P.system == SYS_LORENZ_RK4) launch_basins_pairs<Lorenz>(P, O, l.block, st);
        else if (P.system == SYS_ROSSLER_RK4) launch_basins_pairs<Rossler>(P, O, l.block, st);
        else launch_basins_pairs<Chen>(P, O, l.block, st);
        return cudaGetLastError();
    }
#define CALL(S)                                                              \
    (P.preScaller == 1 ? launch_basins_points<S, true>(P, O, l.block, state, st)    \
                       : launch_basins_points<S, false>(P, O, l.block, state, st))
    CHAOS_SYSTEM_SWITCH(P.system, CALL)
#undef CALL
    return cudaGetLastError();
}

}  // namespace chaos
