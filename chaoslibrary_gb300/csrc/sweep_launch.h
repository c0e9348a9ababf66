// Launch shapes of the FP32 sweeps (kern_f32.cu decides those of the
// bifurcation and basins sweeps, kern_f32_basins.cu shares them) and of the
// FP32 and float-float LLE maps.
#pragma once

#include <algorithm>

#include "launch.h"
#include "systems.h"

namespace chaos {

constexpr int kSweepBlock = 128;  // default block
constexpr int kMaxBlock = 256;    // largest block a tuned launch may use

inline unsigned grid_of(long long threads, int block) { return (unsigned)((threads + block - 1) / block); }

// SMs of the process's first device.
inline long long sm_count() {
    static const long long sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return (long long)std::max(n, 1);
    }();
    return sms;
}

// Blocks of a map's kernel that run one point per thread, before those that run
// two (blocks of kSweepBlock threads). A pair block holds twice the points at
// 1.65 to 1.9 times the time of a single one, so pairs win -- unless the
// points fill an odd number of rows of kSweepBlock per SM: then the pairs' last
// row would be half empty, and one row runs single. It comes first: the
// schedulers favour their oldest warps, and a single block behind pair blocks
// waited until they were done. FP32 Lorenz map, all single / all pairs / this
// rule: one row 0.21 / 0.31 / 0.20 ms, three 0.50 / 0.56 / 0.46, five 0.80 /
// 0.81 / 0.71, seven 1.10 / 1.06 / 0.96 (float-float 1.92 / 2.11 / 1.88), nine
// 1.40 / 1.30 / 1.30. Not where the pairs behind the singles all but fill their
// rows: then some SM gets one more of them than its share, and the map takes as
// long as in pairs alone (three rows: 151 of 152 pair blocks 0.91 ms, spectrum of
// Lorenz, 152 1.16; five: 292 of 304 1.45, 294 1.70; seven: 444 of 456 1.99, 446
// 2.24; the LLE maps alike).
constexpr long long kMixedRows = 7;
inline unsigned single_blocks(long long n) {
    const long long row = kSweepBlock * sm_count(), rows = (n + row - 1) / row;
    if (rows % 2 == 0 || rows > kMixedRows) return 0;
    const long long pairs = n > row ? grid_of((n - row + 1) / 2, kSweepBlock) : 0;
    const long long spare = rows / 2 * sm_count() - pairs;
    if (rows > 1 && spare < (rows == 3 ? 1 : sm_count() / 12)) return 0;
    return grid_of(std::min(n, row), kSweepBlock);
}
// Grid of such a kernel.
inline unsigned mixed_grid(long long n, unsigned singles) {
    const long long left = n - (long long)kSweepBlock * singles;
    return singles + (left > 0 ? grid_of((left + 1) / 2, kSweepBlock) : 0u);
}
// The (first) point of a thread of such a kernel, and whether it has two.
__device__ __forceinline__ long long mixed_point(unsigned singles, bool& pair) {
    pair = blockIdx.x >= singles;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    return pair ? 2 * t - (long long)singles * blockDim.x : t;
}

struct Launch {
    int form;  // 1 one point per thread, 2 packed pairs
    int block;
};
Launch sweep_launch(const SweepParams& P, bool basins);

#define CHAOS_SYSTEM_SWITCH(sys, CALL) \
    switch (sys) {                     \
        case SYS_LORENZ_RK4: CALL(SYS_LORENZ_RK4); break; \
        case SYS_ROSSLER_RK4: CALL(SYS_ROSSLER_RK4); break; \
        case SYS_CHEN_RK4: CALL(SYS_CHEN_RK4); break; \
        case SYS_CHAMELEON: CALL(SYS_CHAMELEON); break; \
        case SYS_ROSSLER_CD: CALL(SYS_ROSSLER_CD); break; \
        case SYS_SIN3: CALL(SYS_SIN3); break; \
        case SYS_SIN2: CALL(SYS_SIN2); break; \
        case SYS_MEMRISTOR: CALL(SYS_MEMRISTOR); break; \
        default: return cudaErrorInvalidValue; \
    }

}  // namespace chaos
