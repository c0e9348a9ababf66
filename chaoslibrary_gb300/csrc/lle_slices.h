// FP32 and float-float LLE maps and spectra in slices of the horizon.
//
// A map runs for as long as its fullest SM: in pairs, whole pair rows of
// 2 * kSweepBlock points per SM, however few SMs have work in the last one. So
// where the points end not far past a row, a launch runs only as many blocks as
// fill the SMs evenly, for a slice of the horizon, and the blocks of points
// ("jobs") take turns from launch to launch, their states in scratch in between.
// Measured at once / in slices: float-float Rossler, 5,510 steps, 1.05 rows of
// kSweepBlock points per SM 2.55 / 1.81 ms, 2.1 rows 3.91 / 2.88, 4.2 rows 6.37 /
// 5.50, 8.2 rows 12.3 / 10.7; FP32 Lorenz, 50,500 steps, 1.05 rows 6.23 / 4.13
// ms, 2.1 rows 9.47 / 6.94, 3.39 rows (257^2 points) 11.66 / 11.11; spectrum of
// Lorenz, 10,500 steps, 1.05 rows 3.05 / 1.79 ms, 4.2 rows 7.00 / 6.03.
// Slices are separate launches on purpose: with the turns taken from a queue by
// resident blocks, jobs held by a young warp of a full SM hardly moved (the
// schedulers favour the oldest warps) and the maps took 1.1 to 1.8 times as long.
#pragma once

#include "engine.cuh"
#include "sweep_launch.h"

namespace chaos {

constexpr int kRowsBeyond = 14;

// What a map's time is made of, in units of what a further row costs the
// kernel that runs it at once.
struct SliceCost {
    double once;        // at once: R rows take R + once
    double row, fixed;  // in slices: row * R + fixed
    double single;      // in slices: one row, a point per thread
    double twin;        // cost of a step with the twins, in transient steps
    int blocks;         // Benettin blocks a slice has a multiple of
    double ns;          // the unit, for one transient step
    int residentRows;   // rows of pairs an SM holds
    int singleRows;     // up to so many rows a map at once runs one point per thread
    constexpr int mostRows() const { return residentRows + kRowsBeyond; }  // of a map that may run in slices
};
// From runs of 1 to 20 rows of the three RK4 systems. At once a row more takes
// 0.287 ms (FP32 Lorenz, 5,500 steps), 0.334 (float-float Rossler, 1,510 steps),
// 0.271 (spectrum, 2,510 steps); a slice kernel's row of FP32 costs more than the
// 56-register kernel's. Slices against one launch, each of the three systems in each
// of the three kernels, 31 sizes from 1.05 to 20.1 rows: 0.71 to 0.99 of the time
// where slices run, but for 1.00 and 1.01 (FP32 at 3.4 rows), 1.01 (spectrum of
// Rossler at 11) -- Chen, whose kernels take other registers, 0.71 to 0.99. residentRows are those of the registers they take, and a
// map of kRowsBeyond more has enough rows not to feel the last one.
constexpr SliceCost kSliceLle{0.36, 1.06, 0.22, 1.48, 2.0, 1, 27.0, 8, 0};
constexpr SliceCost kSliceFF{0.08, 1.0, 0.08, 1.36, 1.1, 1, 208.0, 4, 0};
constexpr SliceCost kSliceSpectrum{0.33, 0.99, 0.29, 1.34, 4.0, kLleGroup, 31.8, 6, 3};
constexpr double kLaunchNs = 8000;  // a launch's start and end, about
constexpr int kMaxSlices = 64;

// jobs == 0: the map runs in one launch. The horizon is counted in units of
// unit transient steps or of the Benettin blocks that cost as much, so that the
// slices of one launch are equally long.
struct SlicePlan {
    int jobs, slices, perLaunch, points;  // points per thread: a job has points * kSweepBlock
    int unit, blocks;                     // of a unit
    int transient, units;                 // units of the transient, and of a slice
    size_t words(int perThread) const { return (size_t)jobs * perThread * kSweepBlock; }
};

inline SlicePlan slice_plan(const LleParams& L, const SliceCost& k) {
    SlicePlan best{};
    const double rows = (double)L.nPoints / (double)(kSweepBlock * sm_count());
    if (rows <= 1.0 || rows > k.mostRows()) return best;
    const long long unit = (long long)(k.twin * L.ntp * k.blocks + 0.5);
    if (unit > 1000000) return best;
    const long long transient = (L.trans + unit - 1) / unit;
    const long long total = transient + ((long long)L.calcBlocks + k.blocks) / k.blocks;
    // one launch: rows of single points, whole pair rows, or an odd number of rows (single_blocks)
    const double whole = std::ceil(rows), even = 2.0 * std::ceil(whole / 2.0) + k.once;
    const double once = whole <= k.singleRows ? whole + 0.27
                        : single_blocks(L.nPoints) ? std::min(even, whole + k.once + 0.16) : even;
    // slices have to promise 3 %: what the model is off by
    double least = 0.97 * once * (double)total * (double)unit * k.ns;
    const int rowsMost = std::min((int)rows, k.residentRows);
    for (int R : {1, rowsMost & ~1}) {
        if (R < 1) continue;
        const int points = R == 1 ? 1 : 2;
        const long long jobs = grid_of((L.nPoints + points - 1) / points, kSweepBlock);
        const long long per = sm_count() * (R == 1 ? 1 : R / 2);
        const double unitNs = (R == 1 ? k.single : k.row * R + k.fixed) * (double)unit * k.ns;
        for (long long q = 2; q <= kMaxSlices && q <= total; ++q) {
            const long long units = (total + q - 1) / q, slices = (total + units - 1) / units;
            const double t = (double)((jobs * slices + per - 1) / per) * ((double)units * unitNs + kLaunchNs);
            if (t >= least) continue;
            least = t;
            best = {(int)jobs, (int)slices, (int)per, points, (int)unit, k.blocks, (int)transient, (int)units};
        }
    }
    return best;
}

// A job's part of a launch.
struct Slice {
    int job;
    int t0, t1, b0, b1;  // transient steps and Benettin blocks
    bool first, last;
    // turn: slices of all jobs in order, slice by slice
    __device__ __forceinline__ Slice(const SlicePlan& plan, const LleParams& L, long long turn) {
        const int slice = (int)(turn / plan.jobs);
        job = (int)(turn - (long long)slice * plan.jobs);
        first = slice == 0;
        last = slice + 1 == plan.slices;
        place(plan, L, slice, t0, b0);
        place(plan, L, slice + 1, t1, b1);
    }
    __device__ __forceinline__ static void place(const SlicePlan& plan, const LleParams& L, int slice, int& t, int& b) {
        const long long at = (long long)slice * plan.units;
        t = (int)min(at * plan.unit, (long long)L.trans);
        b = (int)min(max(at - plan.transient, 0LL) * plan.blocks, (long long)L.calcBlocks + 1);
    }
};

// Words of a thread's state, word i at i * kSweepBlock.
struct StateWords {
    float* at;
    bool save;
    __device__ __forceinline__ void word(float& v) {
        if (save) *at = v;
        else v = *at;
        at += kSweepBlock;
    }
    __device__ __forceinline__ void word(P2& v) {
        word(v.v.x);
        word(v.v.y);
    }
    __device__ __forceinline__ void word(FF<float>& v) {
        word(v.hi);
        word(v.lo);
    }
    __device__ __forceinline__ void word(FF<P2>& v) {
        word(v.hi);
        word(v.lo);
    }
    __device__ __forceinline__ void word(int& v) {
        float f = __int_as_float(v);
        word(f);
        v = __float_as_int(f);
    }
    __device__ __forceinline__ void word(double& v) {
        int lo = __double2loint(v), hi = __double2hiint(v);
        word(lo);
        word(hi);
        v = __hiloint2double(hi, lo);
    }
    template <class T, int N> __device__ __forceinline__ void word(T (&v)[N]) {
#pragma unroll
        for (int i = 0; i < N; ++i) word(v[i]);
    }
};

// One slice of the jobs whose turn it is: from turn on, a job per block.
// results: doubles per point in out.
template <class Point>
__device__ __forceinline__ void run_slice_of(const LleParams& L, const SlicePlan& plan, const Slice& s, float* state,
                                             double* out, int results) {
    const long long o = Point::kPoints * ((long long)s.job * kSweepBlock + threadIdx.x);
    if (o >= L.nPoints) return;
    const bool two = Point::kPoints == 2 && o + 1 < L.nPoints;
    Point z(L, L.pBegin + o, L.pBegin + (two ? o + 1 : o));
    float* mine = state + (size_t)s.job * Point::kWords * kSweepBlock + threadIdx.x;
    if (!s.first) {
        StateWords io{mine, false};
        z.words(io);
    }
    z.transient(s.t1 - s.t0);
    z.blocks(L, s.b0, s.b1);
    if (s.last) {
        double* outp = out + results * o;
        z.result(L, outp, two ? outp + results : nullptr);
    } else {
        StateWords io{mine, true};
        z.words(io);
    }
}

// Both forms in one kernel, as in the kernels that run a map at once: compiled
// alone, with no register need of its own, the float-float point was scheduled
// for 56 registers and took 1.7 times as long.
template <class Pair, class Point>
__device__ __forceinline__ void run_slice(const LleParams& L, const SlicePlan& plan, long long turn, float* state,
                                          double* out, int results) {
    const Slice s(plan, L, turn + blockIdx.x);
    if (plan.points == 2) run_slice_of<Pair>(L, plan, s, state, out, results);
    else run_slice_of<Point>(L, plan, s, state, out, results);
}

template <class K>
void launch_slices(const SlicePlan& plan, K* kernel, const LleParams& L, double* out, float* state, cudaStream_t st) {
    const long long turns = (long long)plan.jobs * plan.slices;
    for (long long t = 0; t < turns; t += plan.perLaunch) {
        kernel<<<(unsigned)std::min<long long>(plan.perLaunch, turns - t), kSweepBlock, 0, st>>>(L, plan, t, state, out);
        note_launch();
    }
}

}  // namespace chaos
