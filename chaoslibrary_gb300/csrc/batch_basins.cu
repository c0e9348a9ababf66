// Group kernels of a batch's basins jobs.
#include "batch_group.cuh"

namespace chaos {

namespace {
// Basins chunks: the RK4 systems as packed pairs (the single sweep's default
// form for large maps), the others one point per thread.
template <int S, bool PRE1>
__device__ __forceinline__ void run_basins_as(const SweepParams& sP, const JobDesc& J, long long b, int cnt) {
    with_component<KnownComponent<S, float>::value && PRE1>(sP.wv, [&](auto wc) {
        if constexpr (S <= SYS_CHEN_RK4) {
#pragma unroll 1
            for (int t = 2 * threadIdx.x; t < cnt; t += 2 * blockDim.x) {
                const long long p = b + t;
                const bool two = t + 1 < cnt;
                basins_pair_point<typename FieldOf<S>::F, PRE1>(sP, J.bas, p, two ? p + 1 : p, p, two ? p + 1 : p,
                                                                two, wc);
            }
        } else {
#pragma unroll 1
            for (int t = threadIdx.x; t < cnt; t += blockDim.x)
                basins_point<S, float, PRE1>(sP, J.bas, b + t, b + t, wc);
        }
    });
}

template <int S>
__device__ __forceinline__ void run_basins(const JobDesc& J, long long b, int cnt) {
    __shared__ SweepParams sP;
    if (threadIdx.x == 0) sP = J.sp;
    __syncthreads();
    if (sP.preScaller == 1) run_basins_as<S, true>(sP, J, b, cnt);
    else run_basins_as<S, false>(sP, J, b, cnt);
}

template <int S> struct BasinsWork {
    static __device__ __forceinline__ void run(const JobDesc& J, long long b, int cnt) { run_basins<S>(J, b, cnt); }
};
}  // namespace

GroupKernel basins_group_kernel(int system) { return group_kernel_of<BasinsWork>(system); }

}  // namespace chaos
