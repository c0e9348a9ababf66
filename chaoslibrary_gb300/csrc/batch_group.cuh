// The persistent group kernels of batched sweeps: one per (kind, system),
// instantiated by batch.cu (LLE maps), batch_bif.cu and batch_basins.cu.
#pragma once

#include "../../include/chaos_gb300.h"
#include "batch.h"
#include "engine.cuh"

namespace chaos {

constexpr int kBatchBlock = 128;

// The group kernels of a batch run at the same time, but an SM holds blocks of
// two kernels only under one split of its memory between L1 and shared memory,
// and left to itself a launch picks the split by the kernel's shared memory and
// residency: blocks of a kernel with 96 registers waited for the SMs of one with
// 104 to fall idle. All of them ask for the most shared memory (their loops
// don't use L1). Six jobs of 84,163 to 841 points 5.68 -> 3.92 ms (a bifurcation
// of 84,163 points alone 2.56, with one of 5,310 beside it 5.38 -> 2.56), nine
// of 60,000 to 600 6.17 -> 5.20, fifteen of 100,000 to 1,000 10.1 either way.
template <class K> void share_sms(K* kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

using GroupKernel = void (*)(const JobDesc*, const Chunk*, int, int*);
GroupKernel bif_group_kernel(int system);
GroupKernel basins_group_kernel(int system);

template <int S> struct FieldOf;
template <> struct FieldOf<SYS_LORENZ_RK4> { using F = Lorenz; };
template <> struct FieldOf<SYS_ROSSLER_RK4> { using F = Rossler; };
template <> struct FieldOf<SYS_CHEN_RK4> { using F = Chen; };

// Persistent kernel of one (kind, system) group: pulls chunks [0, count) of
// the group's range from its counter until none is left. One kernel per
// group keeps each code path's register allocation as small as the
// single-sweep kernel's (a kernel that switched over every kind and system
// would be sized for the largest of them). The RK4 systems' take at most what
// leaves room for five blocks per SM: the bifurcation pairs of Lorenz and Chen
// take 106 and 108 registers unasked, and four blocks of those leave no room for
// one of another group. Nine jobs of 60,000 to 600 points 6.04 -> 5.14 ms, six of
// 100,000 to 1,000 5.27 -> 4.66, twelve of 70,000 to 700 7.29 -> 7.02, fifteen of
// 100,000 to 1,000 9.95 -> 10.02.
template <template <int> class Work, int S>
__global__ void __launch_bounds__(kBatchBlock, S <= SYS_CHEN_RK4 ? 5 : 0) group_kernel(const JobDesc* __restrict__ jobs,
                                                            const Chunk* __restrict__ chunks, int count,
                                                            int* counter) {
    __shared__ int slot;
    for (;;) {
        if (threadIdx.x == 0) slot = atomicAdd(counter, 1);
        __syncthreads();
        const int c = slot;
        __syncthreads();
        if (c >= count) return;
        const Chunk ch = chunks[c];
        const JobDesc& J = jobs[ch.job];
        Work<S>::run(J, ch.begin, ch.count);
    }
}

// The group kernel of a work that every built-in system has.
template <template <int> class Work> GroupKernel group_kernel_of(int system) {
    switch (system) {
        case SYS_LORENZ_RK4: return group_kernel<Work, SYS_LORENZ_RK4>;
        case SYS_ROSSLER_RK4: return group_kernel<Work, SYS_ROSSLER_RK4>;
        case SYS_CHEN_RK4: return group_kernel<Work, SYS_CHEN_RK4>;
        case SYS_CHAMELEON: return group_kernel<Work, SYS_CHAMELEON>;
        case SYS_ROSSLER_CD: return group_kernel<Work, SYS_ROSSLER_CD>;
        case SYS_SIN3: return group_kernel<Work, SYS_SIN3>;
        case SYS_SIN2: return group_kernel<Work, SYS_SIN2>;
        case SYS_MEMRISTOR: return group_kernel<Work, SYS_MEMRISTOR>;
        default: return nullptr;
    }
}

}  // namespace chaos
