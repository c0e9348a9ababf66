// Batched execution of many independent sweeps in one submission.
//
// A batch is a list of jobs (1-D bifurcation, LLE map or basins features;
// any built-in system; uneven sizes and transients). The host cuts every job
// into block-sized chunks of points and groups the chunks by (kind, system),
// each group ordered longest-work-per-point first. Every group gets one
// persistent kernel (resident blocks x SMs, at most one block per chunk)
// that pulls its chunks from a device counter (the work queue); the groups'
// kernels run concurrently on forked streams. A block works on one chunk at
// a time, so every warp runs one job's code path. Each point runs the same
// device function as the single-sweep kernels, so its result does not depend
// on the batch, chunk or block it ran in.
//
// Batches are FP32 (trajectories in FP32 registers, FP64 accumulation) but
// for the float-float LLE jobs, whose group kernel lives with the other FF
// kernels (kern_ff.cu, compiled without contraction); the
// jobs of the RK4 systems run two points per thread (packed FP32x2 lanes),
// the others one. A prepared batch is
// replayed from a captured CUDA graph (counter reset + the group kernels).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../../include/chaos_gb300.h"
#include "batch.h"
#include "capi_internal.h"
#include "batch_group.cuh"

namespace chaos {

namespace {

// The job's parameter block is staged in shared memory for the chunk: read
// from there, the step loop keeps fewer values in registers than when it
// reads them through the global descriptor.
template <class F>
__device__ __forceinline__ void run_lle(const JobDesc& J, long long b, int cnt) {
    __shared__ LleParams sL;
    if (threadIdx.x == 0) sL = J.lp;
    __syncthreads();
    const LleParams& L = sL;
#pragma unroll 1
    for (int t = 2 * threadIdx.x; t < cnt; t += 2 * blockDim.x) {
        const long long p = b + t;
        const bool two = t + 1 < cnt;
        run_point<LlePair<F>>(L, p, two ? p + 1 : p, J.lle + p, two ? J.lle + p + 1 : nullptr);
    }
}

// Chameleon LLE chunks: one point per thread, the twin as the difference of
// chameleon_step_twin (lle_point_twin_chameleon, as the single-sweep kernel).
__device__ __forceinline__ void run_lle_chameleon(const JobDesc& J, long long b, int cnt) {
    __shared__ LleParams sL;
    if (threadIdx.x == 0) sL = J.lp;
    __syncthreads();
#pragma unroll 1
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) J.lle[b + t] = lle_point_twin_chameleon(sL, b + t);
}

template <int S> struct LleWork {
    static __device__ __forceinline__ void run(const JobDesc& J, long long b, int cnt) {
        if constexpr (S <= SYS_CHEN_RK4) run_lle<typename FieldOf<S>::F>(J, b, cnt);
        else run_lle_chameleon(J, b, cnt);
    }
};

__global__ void reset_counters_kernel(int* counters, int n) {
    if ((int)threadIdx.x < n) counters[threadIdx.x] = 0;
}

GroupKernel lle_group_kernel(int system) {
    switch (system) {
        case SYS_LORENZ_RK4: return group_kernel<LleWork, SYS_LORENZ_RK4>;
        case SYS_ROSSLER_RK4: return group_kernel<LleWork, SYS_ROSSLER_RK4>;
        case SYS_CHEN_RK4: return group_kernel<LleWork, SYS_CHEN_RK4>;
        case SYS_CHAMELEON: return group_kernel<LleWork, SYS_CHAMELEON>;
        default: return nullptr;
    }
}

GroupKernel group_kernel_for(int kind, int system) {
    switch (kind) {
        case CHAOS_JOB_BIF1D: return bif_group_kernel(system);
        case CHAOS_JOB_BASINS: return basins_group_kernel(system);
        case CHAOS_JOB_LLE2D: return lle_group_kernel(system);
        default: return nullptr;
    }
}

}  // namespace

// Dynamic shared memory of a group kernel: the sample windows of its threads'
// trajectories (two for the RK4 systems).
static size_t group_shared_bytes(int kind, int system) {
    if (kind != CHAOS_JOB_BIF1D && kind != CHAOS_JOB_BASINS) return 0;
    return system <= SYS_CHEN_RK4 ? Window<2>::bytes(kBatchBlock) : Window<1>::bytes(kBatchBlock);
}

int batch_block_size() { return kBatchBlock; }

int group_resident_blocks(int kind, int system, int device) {
    if (kind == CHAOS_JOB_LLE2D_FF32) return group_ff_resident_blocks(system, device);
    GroupKernel k = group_kernel_for(kind, system);
    if (!k) return 0;
    share_sms(k);
    int perSm = 0, sms = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k, kBatchBlock, group_shared_bytes(kind, system));
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return std::max(perSm, 1) * std::max(sms, 1);
}

cudaError_t reset_counters(int* counters, int n, cudaStream_t st) {
    reset_counters_kernel<<<1, 32, 0, st>>>(counters, n);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_group(int kind, int system, const JobDesc* jobs, const Chunk* chunks, int count, int* counter,
                         int gridBlocks, cudaStream_t st) {
    if (kind == CHAOS_JOB_LLE2D_FF32) return launch_group_ff(system, jobs, chunks, count, counter, gridBlocks, st);
    GroupKernel k = group_kernel_for(kind, system);
    if (!k) return cudaErrorInvalidValue;
    if (count <= 0) return cudaSuccess;
    share_sms(k);
    k<<<gridBlocks, kBatchBlock, group_shared_bytes(kind, system), st>>>(jobs, chunks, count, counter);
    note_launch();
    return cudaGetLastError();
}

}  // namespace chaos
