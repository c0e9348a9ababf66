// Transients of the FP32 sweeps that run one point per thread, in slices.
//
// As with the LLE maps (lle_slices.h), a sweep takes as long as its fullest SM:
// T(R) for R rows of kSweepBlock points per SM, with R rounded up. Where the
// points end not far past a row the transient runs in launches of as many
// blocks as fill the SMs evenly, each for a slice of the steps, the blocks of
// points taking turns with their states in scratch; the sweep kernel then
// starts from those states (a last step before it, for the fixed-point test).
#pragma once

#include "engine.cuh"
#include "sweep_launch.h"

namespace chaos {

// Time of R rows in units of ns per step, from transients of 20,000 steps, 1 to
// 16 full rows: Lorenz 0.69, 1.12, 1.72, 2.19, 2.75, 3.25 ms, 8 rows 4.31, 16
// 8.6 (Rossler 4 % less); Chameleon, which waits for its cosine, 1.76 (1.87 in
// slices), 1.97, 2.30, 2.53, 3.20, 3.82 ms, 8 rows 4.82, 16 8.9.
// At once / in slices, whole sweeps: Lorenz, transient 100,000 and 10,000 recorded
// steps, 1.05 rows 6.21 / 4.36 ms, 2.1 rows 9.47 / 6.84, 4.2 rows 15.3 / 13.2, 8.2
// rows 26.9 / 25.2; Chameleon 4.2 rows 17.6 / 15.5, 4.63 rows (300^2) 17.6 / 16.9.
constexpr double kTransientNs = 26.0;
inline double transient_time(int system, int rows) {
    if (system != SYS_CHAMELEON) return rows == 1 ? 1.3 : rows + (rows % 2 ? 0.22 : 0.12);
    constexpr double few[5] = {0.0, 3.60, 3.79, 4.43, 4.87};
    return rows <= 4 ? few[rows] : 0.97 * rows + 1.4;
}
constexpr double kTransientLaunchNs = 8000;  // a launch's start and end, about
constexpr int kTransientRows = 16;           // more rows hardly feel the last one (and RK4 sweeps run in pairs)
constexpr int kTransientSlices = 64;

// jobs == 0: no slices.
struct TransientPlan {
    int jobs, perLaunch, slices, steps;  // steps of a slice
    int total;                           // steps of the transient that are sliced
    size_t bytes() const { return (size_t)jobs * kSweepBlock * sizeof(float4); }
};

// The sliced steps of a sweep's transient: all but the last for the
// bifurcation, which compares the last two states.
inline TransientPlan transient_plan(const SweepParams& P, bool basins) {
    TransientPlan best{};
    const long long row = kSweepBlock * sm_count();
    if (P.nPoints <= row || P.nPoints > kTransientRows * row || P.sweepStep ||
        !(P.system <= SYS_CHEN_RK4 || P.system == SYS_CHAMELEON))
        return best;
    const Launch l = sweep_launch(P, basins);
    const int total = basins ? P.S : P.S - 1;
    if (l.form != 1 || l.block != kSweepBlock || total < 256) return best;
    const long long jobs = grid_of(P.nPoints, kSweepBlock);
    double least = 0.97 * transient_time(P.system, (int)((P.nPoints + row - 1) / row)) * total * kTransientNs;
    for (int R = 1; R <= (int)(P.nPoints / row); ++R) {
        const long long per = R * sm_count();
        for (int q = 2; q <= kTransientSlices; ++q) {
            const int steps = ((total + q - 1) / q + 7) / 8 * 8, slices = (total + steps - 1) / steps;
            const double t = (double)((jobs * slices + per - 1) / per) *
                             (steps * transient_time(P.system, R) * kTransientNs + kTransientLaunchNs);
            if (t >= least) continue;
            least = t;
            best = {(int)jobs, (int)per, slices, steps, total};
        }
    }
    return best;
}

// A slice of the jobs whose turn it is, a block each: x and flag (1, or 0 once
// diverged) of point job * kSweepBlock + threadIdx.x in state.
template <int S, int W, bool Basins>
__global__ void __launch_bounds__(kSweepBlock) transient_slice_kernel_f32(SweepParams P, TransientPlan plan,
                                                                          long long turn, float4* state) {
    static_assert(Traits<S>::NX == 3, "three state components");
    const int slice = (int)((turn + blockIdx.x) / plan.jobs);
    const long long o = (turn + blockIdx.x - (long long)slice * plan.jobs) * kSweepBlock + threadIdx.x;
    if (o >= P.nPoints) return;
    float x[3], a[Traits<S>::NA];
    load_point<S, float>(P, P.pBegin + o, x, a);
    bool flag = true;
    if (slice > 0) {
        const float4 v = state[o];
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
        flag = v.w != 0.f;
    }
    const StepCtx<float> c((float)P.h);
    const Component<W> wc{P.wv};
    const int n = min(plan.steps, plan.total - slice * plan.steps);
    int s = 0;
    constexpr int K = kTransientBlock;
    for (; flag && s + K <= n; s += K) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
            step<S>(x, a, c);
            if (!Basins && bif_diverged(wc.template of<3>(x), P)) flag = false;
        }
    }
    for (; flag && s < n; ++s) {
        step<S>(x, a, c);
        if (!Basins && bif_diverged(wc.template of<3>(x), P)) flag = false;
    }
    state[o] = make_float4(x[0], x[1], x[2], flag ? 1.f : 0.f);
}

template <int S, int W, bool Basins>
void launch_transient(const TransientPlan& plan, const SweepParams& P, float4* state, cudaStream_t st) {
    const long long turns = (long long)plan.jobs * plan.slices;
    for (long long t = 0; t < turns; t += plan.perLaunch) {
        transient_slice_kernel_f32<S, W, Basins>
            <<<(unsigned)std::min<long long>(plan.perLaunch, turns - t), kSweepBlock, 0, st>>>(P, plan, t, state);
        note_launch();
    }
}

}  // namespace chaos
