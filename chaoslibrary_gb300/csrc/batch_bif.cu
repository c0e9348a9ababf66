// Group kernels of a batch's bifurcation jobs.
#include "batch_group.cuh"

namespace chaos {

namespace {
// Bifurcation chunks: the RK4 systems as packed pairs (chunks of two blocks'
// worth of points), the others one point per thread.
template <int S>
__device__ __forceinline__ void run_bif(const JobDesc& J, long long b, int cnt) {
    __shared__ SweepParams sP;
    if (threadIdx.x == 0) sP = J.sp;
    __syncthreads();
    with_component<KnownComponent<S, float>::value>(sP.wv, [&](auto wc) {
        if constexpr (S <= SYS_CHEN_RK4) {
#pragma unroll 1
            for (int t = 2 * threadIdx.x; t < cnt; t += 2 * blockDim.x) {
                const long long p = b + t;
                const bool two = t + 1 < cnt;
                bif_pair_point<typename FieldOf<S>::F>(sP, J.bif, p, two ? p + 1 : p, p, two ? p + 1 : p, two, wc);
            }
        } else {
#pragma unroll 1
            for (int t = threadIdx.x; t < cnt; t += blockDim.x) bif_point<S, float>(sP, J.bif, b + t, b + t, wc);
        }
    });
}

template <int S> struct BifWork {
    static __device__ __forceinline__ void run(const JobDesc& J, long long b, int cnt) { run_bif<S>(J, b, cnt); }
};
}  // namespace

GroupKernel bif_group_kernel(int system) { return group_kernel_of<BifWork>(system); }

}  // namespace chaos
