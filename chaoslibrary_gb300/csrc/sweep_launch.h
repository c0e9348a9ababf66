// Launch shapes of the FP32 bifurcation and basins sweeps (kern_f32.cu decides
// them, kern_f32_basins.cu shares them).
#pragma once

#include "launch.h"
#include "systems.h"

namespace chaos {

constexpr int kSweepBlock = 128;  // default block
constexpr int kMaxBlock = 256;    // largest block a tuned launch may use

inline unsigned grid_of(long long threads, int block) { return (unsigned)((threads + block - 1) / block); }

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
