// FP64 kernels: the reference's arithmetic, one rounding per written
// operation. This translation unit is compiled with --fmad=false, so a*b+c
// stays two roundings unless the source calls fma(); together with IEEE
// division and square root the FP64 sweeps reproduce the CPU oracle bit for
// bit. Also holds the reference-semantics kernels that run on caller arrays
// (peak finder, per-point dbscan of the 2-D bifurcation).
#include <algorithm>
#include <climits>

#include "engine.cuh"
#include "legacy_lle.cuh"
#include "sweep_launch.h"
#include "team.cuh"

namespace chaos {

namespace {
constexpr int kBlock = 128;
// Blocks of the sweep kernels: one warp. A warp's FP64 instruction occupies
// its pipe for about 64 cycles and one SM issues one every 16 to 18, so an SM
// with w warps takes time proportional to w from four on, and what counts is
// that no SM gets a warp more than another. Measured (25,000 Lorenz steps, a
// 150^2 basins map, 704 warps on 152 SMs): blocks of four warps 81.4 ms (two
// blocks on some SMs), of one warp 60.7 ms; a 100^2 Rossler LLE map 85.7 -> 75.5 ms.
constexpr int kSweep = 32;

// Legacy: the legacy library's per-point loop (P.legacyLoop != 0).
template <int S, bool Legacy>
__global__ void __launch_bounds__(kSweep) bif_kernel(SweepParams P, BifOut O) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= P.nPoints) return;
    if constexpr (Legacy) bif_point_legacy<S>(P, O, P.pBegin + o, o);
    else bif_point<S, double>(P, O, P.pBegin + o, o, Component<-1>{P.wv});
}

// Bifurcation points list[0, count), result row k for list[k].
template <int S, bool Legacy>
__global__ void __launch_bounds__(kSweep) bif_list_kernel(SweepParams P, BifOut O, const int* list, int count) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    if constexpr (Legacy) bif_point_legacy<S>(P, O, list[k], k);
    else bif_point<S, double>(P, O, list[k], k, Component<-1>{P.wv});
}

template <int S>
__global__ void __launch_bounds__(kSweep) basins_kernel(SweepParams P, BasinsOut O) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= P.nPoints) return;
    basins_point<S, double, false>(P, O, P.pBegin + o, o, Component<-1>{P.wv});
}

template <int S>
__global__ void __launch_bounds__(kSweep) lle_kernel(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    out[o] = lle_point_full<S, double>(L, L.pBegin + o);
}

// Small sweeps of the RK4 systems, a team of three lanes per trajectory (team.cuh).
template <class F>
__global__ void __launch_bounds__(kSweep) bif_team_kernel(SweepParams P, BifOut O) {
    __shared__ double cols[kTeamColumn * TeamLane::kTeams];
    bif_teams<F>(P, O, cols);
}
template <class F>
__global__ void __launch_bounds__(kSweep) basins_team_kernel(SweepParams P, BasinsOut O) {
    __shared__ double cols[kTeamColumn * TeamLane::kTeams];
    basins_teams<F>(P, O, cols);
}
template <class F, int G>
__global__ void __launch_bounds__(kSweep) lle_team_kernel(LleParams L, double* out) {
    lle_teams<F, G>(L, out);
}
template <class F, int G>
__global__ void __launch_bounds__(kSweep) spectrum_team_kernel(LleParams L, double* out) {
    spectrum_teams<F, G>(L, out);
}

// The legacy library's LLE kernels' scheme (L.legacyLoop).
template <int S>
__global__ void __launch_bounds__(kSweep) lle_legacy_kernel(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    out[o] = lle_point_legacy<S>(L, L.pBegin + o);
}

// The LLE map with the reference's cuRAND twin start (L.twin == 2).
template <int S>
__global__ void __launch_bounds__(kSweep) lle_reftwin_kernel(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    out[o] = lle_point_reftwin<S>(L, L.pBegin + o);
}

// kind 0 / 1: out[p*nx + k] = legacy_twin_draw; kind 2: out[(p*nx + j)*nx + i] = legacy_spectrum_draw
__global__ void legacy_draws_kernel(int kind, long long n, int nx, double* out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long per = kind == 2 ? (long long)nx * nx : nx;
    if (t >= n * per) return;
    const long long p = t / per;
    const int r = (int)(t % per);
    out[t] = kind == 2 ? legacy_spectrum_draw(p, r % nx, r / nx) : legacy_twin_draw(kind, p, r);
}

// Benettin blocks from caller-supplied starting states (the reference's
// semi_result layout, LLE/src/LLECUDA.cu:102-111): point k's row of 2*NX + NA
// values holds the orbit after the transient, the parameters and the twin.
template <int S>
__global__ void __launch_bounds__(kSweep) lle_states_kernel(LleParams L, const double* states, double* out) {
    constexpr int NX = Traits<S>::NX, NA = Traits<S>::NA, W = 2 * NX + NA;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= L.nPoints) return;
    const double* r = states + k * W;
    double x[NX], q[NX], a[NA];
#pragma unroll
    for (int i = 0; i < NX; ++i) {
        x[i] = r[i];
        q[i] = r[NX + NA + i];
    }
#pragma unroll
    for (int i = 0; i < NA; ++i) a[i] = r[NX + i];
    out[k] = lle_benettin_full<S>(L, x, q, a);
}

// Lyapunov spectrum, out[p*SIZE_X + j]
template <int S>
__global__ void __launch_bounds__(kSweep) spectrum_kernel(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    spectrum_point_full<S>(L, L.pBegin + o, out);
}

// The legacy library's spectrum kernel's scheme (L.legacyLoop).
template <int S>
__global__ void __launch_bounds__(kSweep) spectrum_legacy_kernel(LleParams L, double* out) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= L.nPoints) return;
    spectrum_point_legacy<S>(L, L.pBegin + o, out);
}

// FP64 LLE of the points list[0, *count): out[k] (scatter = 0) or out[list[k]]
// (scatter = 1). The same device function as lle_kernel, so a point's value
// is the FP64 map's value bit for bit.
template <int S>
__global__ void __launch_bounds__(kSweep) lle_list_kernel(LleParams L, const int* list, const int* count,
                                                          double* out, int scatter) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= *count) return;
    const int p = list[k];
    const double v = lle_point_full<S, double>(L, p);
    out[scatter ? p : k] = v;
}

// class of an LLE value for the sign re-check: 1 positive, 0 non-positive,
// -1 not finite
__device__ __forceinline__ int lle_class(double v) { return !(fabs(v) <= 1.7976931348623157e308) ? -1 : v > 0.0; }

// warp-aggregated append of p to list (one atomic per warp; list may be null
// to count only)
__device__ __forceinline__ void append(bool take, int p, int* list, int* count) {
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (!m) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (take && list) list[base + __popc(m & ((1u << lane) - 1))] = p;
}

// points whose value is within band of zero or not finite
__global__ void lle_select_kernel(const double* v, long long n, double band, int* list, int* count) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool take = i < n && !(fabs(v[i]) > band);
    append(take, (int)i, list, count);
}

// checked points whose FP64 check disagrees in class with the FP32 value are
// counted in count2 and appended to list2 (when not null); with final = 1
// (the check ran the full horizon) their check value is stored into out.
// Every thread of the grid reaches the warp vote.
__global__ void lle_flip_kernel(const double* v32, const int* list, const int* count, const double* check,
                                int final_, double* out, int* list2, int* count2) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool take = false;
    int p = 0;
    if (k < *count) {
        p = list[k];
        take = lle_class(v32[p]) != lle_class(check[k]);
    }
    append(take, p, list2, count2);
    if (take && final_) out[p] = check[k];
}

template <int S>
__global__ void __launch_bounds__(kBlock) trajectory_kernel(const double* x0, const double* a0, double h, int nSteps,
                                                       double* out, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    trajectory_point<S, double>(x0, a0, h, nSteps, out, t);
}

inline unsigned grid_for(long long n) { return (unsigned)((n + kBlock - 1) / kBlock); }
inline unsigned warps_for(long long n) { return (unsigned)((n + kSweep - 1) / kSweep); }

// Peak finder over caller series (the reference's peakFinderCUDA semantics on
// identical input arrays): one thread streams one series.
__global__ void peak_array_kernel(const double* __restrict__ data, long long nSeries, int len, double h, int cap,
                                  int* counts, double* peaks, double* intervals) {
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nSeries) return;
    const double* d = data + s * (long long)len;
    PeakStream<double> ps;
    ps.init();
    for (int k = 0; k < len; ++k) {
        double val;
        int t;
        if (ps.push(d[k], val, t)) {
            if (ps.n >= 1) {
                const int q = ps.n - 1;
                if (q < cap) {
                    peaks[s * (long long)cap + q] = val;
                    intervals[s * (long long)cap + q] = __dmul_rn((double)(t - ps.tprev), h);
                }
            }
            ps.tprev = t;
            ++ps.n;
        }
    }
    counts[s] = ps.n > 1 ? ps.n - 1 : 0;
}

// Per-point dbscan of the 2-D bifurcation (bifurcationCUDA.cu:516-583), one
// warp per point. The sequential control (new cluster / pop of slot NN-1) is
// uniform across the warp; each expansion pass over k < P-1 is split across
// the lanes, which is exact because pass k only reads and writes entry k.
//
// A label is only ever asked whether it is set, and slot k only ever holds k
// or 0, so a row of at most 1,024 intervals keeps both as bits: bit m of a
// lane's word stands for entry 32 m + lane. A pass visits only the groups of
// 32 that have an unlabelled entry, and the walk stops once every entry below
// the last is labelled: the pops that are left label nothing and the last
// entry, if open, makes one more cluster. A pop of 0 outside the first cluster
// is skipped too, as entry 0 was expanded first and the unlabelled entries
// only get fewer. The distances go by a float copy of the row in shared memory
// unless the error bound of the float difference leaves the limit open: with
// an FP64 subtraction and conversion per pair the FP64 pipe bounded it. 300^2
// points of the Chameleon with 60 intervals each: 2.40 ms with labels and slots
// in scratch, 0.98 ms with the bits, 0.32 ms with the float copy; then issue
// slots bound it (89 % busy, 90,000 rows of 60 intervals 0.14 to 0.33 ms).
constexpr int kDbscanBits = 1024;

// distance < eps of two intervals: the distance is 0 for equal ones (also
// infinite ones) and the float magnitude of the difference otherwise. lim is
// the least float not below eps, which decides like eps for every float.
__device__ __forceinline__ bool interval_near(double a, double b, float lim) {
    const float dist = fabsf((float)(b - a));
    return dist < lim || (isinf(a) && a == b && 0.0f < lim);
}

__device__ __forceinline__ int dbscan_bits(const double* __restrict__ iv, int P, float lim, int lane, float* fv) {
    for (int k = lane; k < P; k += 32) fv[k] = (float)iv[k];
    __syncwarp();
    const int last = P - 1;  // never labelled by a pass
    const int mine = last > lane ? (last - lane + 31) >> 5 : 0;  // entries below the last one in this lane
    unsigned fresh = mine >= 32 ? ~0u : (1u << mine) - 1u;
    const int groups = (last + 31) >> 5;
    unsigned open = groups >= 32 ? ~0u : (1u << groups) - 1u;
    unsigned slots = 0;
    bool lastOpen = true;
    int cluster = 0, nn = 0;
    for (int i = 0; i < P; ++i) {
        if (nn >= 1) {
            const int s = --nn;
            const unsigned word = __shfl_sync(0xffffffffu, slots, s & 31);
            i = (word >> (s >> 5)) & 1u ? s : 0;
            if (lane == (s & 31)) slots &= ~(1u << (s >> 5));
            if (i == 0) continue;
        } else {
            unsigned f = fresh & (~0u << (i >> 5));
            if (lane < (i & 31)) f &= ~(1u << (i >> 5));
            i = __reduce_min_sync(0xffffffffu, f ? ((__ffs((int)f) - 1) << 5) + lane : last);
            if (i == last) {
                if (!lastOpen) break;
                lastOpen = false;
            } else if (lane == (i & 31)) {
                fresh &= ~(1u << (i >> 5));
            }
            ++cluster;
        }
        const float fi = fv[i];
#pragma unroll 3
        for (unsigned o = open; o; o &= o - 1u) {
            const int m = __ffs((int)o) - 1;
            const unsigned bit = 1u << m;
            bool hit = false;
            if (fresh & bit) {
                const int k = (m << 5) + lane;
                const float fk = fv[k], d = fabsf(fk - fi);
                // two conversions, the two differences and the sum below each
                // round by at most 2^-24 of |fi| + |fk|
                const float err = fmaf(fabsf(fi) + fabsf(fk), 0x1p-21f, 0x1p-126f);
                hit = d + err < lim;
                if (!hit && !(d - err >= lim)) hit = interval_near(iv[i], iv[k], lim);
            }
            if (hit) {
                fresh &= ~bit;
                slots |= bit;
            }
            nn += __popc(__ballot_sync(0xffffffffu, hit));
            if (!__any_sync(0xffffffffu, fresh & bit)) open &= ~bit;
        }
        if (!open) {
            cluster += lastOpen;
            break;
        }
    }
    return cluster;
}

// Longer rows: labels and slots in scratch, one int an entry.
__device__ __forceinline__ int dbscan_scratch(const double* __restrict__ iv, int P, float lim, int lane, int* lab,
                                              int* slot) {
    for (int k = lane; k < P; k += 32) { lab[k] = 0; slot[k] = 0; }
    __syncwarp();
    int cluster = 0, nn = 0;
    for (int i = 0; i < P; ++i) {
        bool expand = false;
        if (nn >= 1) {
            i = slot[nn - 1];
            __syncwarp();
            if (lane == 0) slot[nn - 1] = 0;
            --nn;
            expand = true;
        } else if (lab[i] == 0) {
            ++cluster;
            __syncwarp();
            if (lane == 0) lab[i] = cluster;
            expand = true;
        }
        if (expand) {
            __syncwarp();
            const double ivi = iv[i];
            for (int k0 = 0; k0 < P - 1; k0 += 32) {
                const int k = k0 + lane;
                bool hit = false;
                if (k < P - 1 && lab[k] == 0 && interval_near(ivi, iv[k], lim)) {
                    lab[k] = cluster;
                    slot[k] = k;
                    hit = true;
                }
                nn += __popc(__ballot_sync(0xffffffffu, hit));
            }
            __syncwarp();
        }
    }
    return cluster;
}

// Long: the rows of more than kDbscanBits intervals, otherwise the others. A
// kernel of their own, as they live in the L1 cache, which the others' shared
// memory takes room from: 300 rows of up to 3,000 intervals 107 ms with both in
// one kernel, 63 apart; 90,000 of up to 1,200 150 and 134.
template <bool Long>
__global__ void point_dbscan_kernel(const double* __restrict__ intervals, const int* __restrict__ counts, long long n,
                                    int stride, double eps, int* labScratch, int* slotScratch, int* outBase,
                                    const int* outIdx) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= n) return;
    const long long oi = outIdx ? (long long)outIdx[w] : w;  // where this point's label goes
    const int P = counts[w];
    if (Long != (P > kDbscanBits && P <= stride)) return;
    if (P > stride) {  // more intervals than the row holds: reported, not read
        if (lane == 0) outBase[oi] = INT_MIN;
        return;
    }
    if (P <= 1) {  // dbscanCUDA: -1 passes through; dbscan returns 0 for P <= 0 and 1 for P == 1
        if (lane == 0) outBase[oi] = P == -1 ? -1 : (P == 1 ? 1 : 0);
        return;
    }
    const long long row = w * (long long)stride;
    const float lim = __double2float_ru(eps);
    int cluster;
    if constexpr (Long) {
        cluster = dbscan_scratch(intervals + row, P, lim, lane, labScratch + row, slotScratch + row);
    } else {
        extern __shared__ float rows[];  // min(stride, kDbscanBits) a warp
        cluster = dbscan_bits(intervals + row, P, lim, lane, rows + (threadIdx.x >> 5) * min(stride, kDbscanBits));
    }
    if (lane == 0) outBase[oi] = cluster - 1;
}

}  // namespace

bool system_supported(int system) {
    return (system >= 0 && system < SYS_COUNT) || (system == SYS_USER && user_system_available());
}
int launch_block_size() { return kBlock; }

// Which sweeps run in teams, by points per SM. Their time grows with the
// points, that of the kernels with a point per thread with whole warps per SM
// (flat up to three, 128 points 7 % more, 160 points 1.47 times). Measured,
// point per thread against teams, Lorenz, 4,000 steps: 1,000 points 6.47 /
// 3.24 ms, 9,000 6.46 / 3.66, 15,200 6.90 / 5.58, 18,240 (120 per SM) 6.90 /
// 6.63, 19,456 (128) 6.90 / 7.48, 22,800 (150) 9.49 / 8.28; a 150^2 basins map
// (25,000 steps) 60.7 / 47.3 ms. LLE maps (with the blocks' norms and logs,
// which every lane of a team takes), 3,020 steps of orbit and twin, Rossler
// 40^2 7.12 / 4.24 ms, 100^2 7.12 / 6.10, 110^2 (80 per SM) 7.12 / 6.95, 116^2
// 7.12 / 8.23; orbit and twin in a team each 40^2 2.62 ms, 77^2 (39 per SM)
// 4.33 against 4.41 in one team, 90^2 5.95 against 5.32.
long long sm_points(long long perSm) { return perSm * sm_count(); }
bool team_sweep(long long n) {
    return n <= sm_points(120) || (n > sm_points(128) && n <= sm_points(160));
}
bool team_lle(long long n) { return n <= sm_points(80); }
bool split_lle(long long n) { return n <= sm_points(40); }
// Spectra (the three twins and the Gram-Schmidt beside the orbit), 500 steps,
// point per thread / four trajectories a team / a team each, Lorenz: up to 10
// points per SM 2.99 / 1.62 / 0.58 to 0.64 ms, 16 2.99 / 1.62 / 0.89, 26 2.99 /
// 1.62 / 1.46, 32 2.99 / 1.69 / 1.74, 60 2.99 / 1.99, 80 2.99 / 2.54, 90 2.99 /
// 3.00; Rossler 26 2.55 / 1.59 / 1.51, 70 2.55 / 2.32, 80 2.55 / 2.63; Chen 80
// 3.21 / 3.03, 90 3.22 / 3.56.
bool team_spectrum(long long n) { return n <= sm_points(76); }
bool split_spectrum(long long n) { return n <= sm_points(28); }
inline unsigned team_blocks(long long n, int perWarp) { return (unsigned)((n + perWarp - 1) / perWarp); }

#define CHAOS_RK4_SWITCH(sys, CALL)                  \
    switch (sys) {                                   \
        case SYS_LORENZ_RK4: CALL(Lorenz); break;    \
        case SYS_ROSSLER_RK4: CALL(Rossler); break;  \
        case SYS_CHEN_RK4: CALL(Chen); break;        \
        default: return cudaErrorInvalidValue;       \
    }

cudaError_t launch_bif_f64(const SweepParams& P, const BifOut& O, cudaStream_t st) {
    if (P.nPoints <= 0) return cudaSuccess;
    if (P.system <= SYS_CHEN_RK4 && !P.legacyLoop && !P.sweepStep && team_sweep(P.nPoints)) {
#define CALL(F) bif_team_kernel<F><<<team_blocks(P.nPoints, TeamLane::kTeams), kSweep, 0, st>>>(P, O)
        CHAOS_RK4_SWITCH(P.system, CALL)
#undef CALL
        note_launch();
        return cudaGetLastError();
    }
#define CALL(S)                                                             \
    {                                                                       \
        if (P.legacyLoop) bif_kernel<S, true><<<warps_for(P.nPoints), kSweep, 0, st>>>(P, O); \
        else bif_kernel<S, false><<<warps_for(P.nPoints), kSweep, 0, st>>>(P, O); \
        note_launch();                                                      \
    }
    CHAOS_SYSTEM_SWITCH(P.system, CALL)
#undef CALL
    return cudaGetLastError();
}

cudaError_t launch_basins_f64(const SweepParams& P, const BasinsOut& O, cudaStream_t st) {
    if (P.nPoints <= 0) return cudaSuccess;
    if (P.system <= SYS_CHEN_RK4 && team_sweep(P.nPoints)) {
#define CALL(F) basins_team_kernel<F><<<team_blocks(P.nPoints, TeamLane::kTeams), kSweep, 0, st>>>(P, O)
        CHAOS_RK4_SWITCH(P.system, CALL)
#undef CALL
        note_launch();
        return cudaGetLastError();
    }
#define CALL(S) (basins_kernel<S><<<warps_for(P.nPoints), kSweep, 0, st>>>(P, O), note_launch())
    CHAOS_SYSTEM_SWITCH(P.system, CALL)
#undef CALL
    return cudaGetLastError();
}

cudaError_t launch_lle_f64(const LleParams& L, double* out, cudaStream_t st) {
    if (L.nPoints <= 0) return cudaSuccess;
    if (L.system <= SYS_CHEN_RK4 && !L.legacyLoop && L.twin != 2 && team_lle(L.nPoints)) {
        const bool split = split_lle(L.nPoints);
#define CALL(F)                                                                                                 \
    (split ? lle_team_kernel<F, 2><<<team_blocks(L.nPoints, TeamLane::kTeams / 2), kSweep, 0, st>>>(L, out)     \
           : lle_team_kernel<F, 1><<<team_blocks(L.nPoints, TeamLane::kTeams), kSweep, 0, st>>>(L, out))
        CHAOS_RK4_SWITCH(L.system, CALL)
#undef CALL
        note_launch();
        return cudaGetLastError();
    }
#define CALL(S)                                                               \
    {                                                                         \
        if (L.legacyLoop) lle_legacy_kernel<S><<<warps_for(L.nPoints), kSweep, 0, st>>>(L, out); \
        else if (L.twin == 2) lle_reftwin_kernel<S><<<warps_for(L.nPoints), kSweep, 0, st>>>(L, out); \
        else lle_kernel<S><<<warps_for(L.nPoints), kSweep, 0, st>>>(L, out); \
        note_launch();                                                        \
    }
    CHAOS_SYSTEM_SWITCH(L.system, CALL)
#undef CALL
    return cudaGetLastError();
}

cudaError_t launch_legacy_draws(int kind, long long n, int nx, double* out, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    legacy_draws_kernel<<<grid_for(n * (kind == 2 ? (long long)nx * nx : nx)), kBlock, 0, st>>>(kind, n, nx, out);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_lle_states_f64(const LleParams& L, const double* states, double* out, cudaStream_t st) {
    if (L.nPoints <= 0) return cudaSuccess;
#define CALL(S) (lle_states_kernel<S><<<warps_for(L.nPoints), kSweep, 0, st>>>(L, states, out), note_launch())
    CHAOS_SYSTEM_SWITCH(L.system, CALL)
#undef CALL
    return cudaGetLastError();
}

cudaError_t launch_spectrum_f64(const LleParams& L, double* out, cudaStream_t st) {
    if (L.nPoints <= 0) return cudaSuccess;
    if (!L.legacyLoop && L.system <= SYS_CHEN_RK4 && team_spectrum(L.nPoints)) {
        const bool split = split_spectrum(L.nPoints);
#define CALL(F)                                                                                         \
    (split ? spectrum_team_kernel<F, 4><<<team_blocks(L.nPoints, 2), kSweep, 0, st>>>(L, out)           \
           : spectrum_team_kernel<F, 1><<<team_blocks(L.nPoints, TeamLane::kTeams), kSweep, 0, st>>>(L, out))
        CHAOS_RK4_SWITCH(L.system, CALL)
#undef CALL
        note_launch();
        return cudaGetLastError();
    }
#define CALL(S)                                                                    \
    {                                                                              \
        if (L.legacyLoop) spectrum_legacy_kernel<S><<<warps_for(L.nPoints), kSweep, 0, st>>>(L, out); \
        else spectrum_kernel<S><<<warps_for(L.nPoints), kSweep, 0, st>>>(L, out); \
        note_launch();                                                             \
    }
    CHAOS_SYSTEM_SWITCH(L.system, CALL)
#undef CALL
    return cudaGetLastError();
}

cudaError_t launch_bif_list_f64(const SweepParams& P, const BifOut& O, const int* list, int count, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
#define CALL(S)                                                                       \
    {                                                                                 \
        if (P.legacyLoop) bif_list_kernel<S, true><<<warps_for(count), kSweep, 0, st>>>(P, O, list, count); \
        else bif_list_kernel<S, false><<<warps_for(count), kSweep, 0, st>>>(P, O, list, count); \
        note_launch();                                                                \
    }
    CHAOS_SYSTEM_SWITCH(P.system, CALL)
#undef CALL
    return cudaGetLastError();
}

// indices of the points whose kept-peak count exceeds cap
__global__ void overflow_select_kernel(const int* counts, long long n, int cap, int* list, int* count) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    append(i < n && counts[i] > cap, (int)i, list, count);
}

cudaError_t launch_overflow_select(const int* counts, long long n, int cap, int* list, int* count, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    overflow_select_kernel<<<grid_for(n), kBlock, 0, st>>>(counts, n, cap, list, count);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_lle_select(const double* v, long long n, double band, int* list, int* count, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    lle_select_kernel<<<grid_for(n), kBlock, 0, st>>>(v, n, band, list, count);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_lle_list_f64(const LleParams& L, const int* list, const int* count, long long maxCount,
                                double* out, bool scatter, cudaStream_t st) {
    if (maxCount <= 0) return cudaSuccess;
#define CALL(S) \
    (lle_list_kernel<S><<<warps_for(maxCount), kSweep, 0, st>>>(L, list, count, out, scatter ? 1 : 0), note_launch())
    CHAOS_SYSTEM_SWITCH(L.system, CALL)
#undef CALL
    return cudaGetLastError();
}

cudaError_t launch_lle_flip(const double* v32, const int* list, const int* count, long long maxCount,
                            const double* check, bool final_, double* out, int* list2, int* count2, cudaStream_t st) {
    if (maxCount <= 0) return cudaSuccess;
    lle_flip_kernel<<<grid_for(maxCount), kBlock, 0, st>>>(v32, list, count, check, final_ ? 1 : 0, out, list2,
                                                            count2);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_peak_finder(const double* data, long long nSeries, int len, double h, int cap, int* counts,
                               double* peaks, double* intervals, cudaStream_t st) {
    if (nSeries <= 0) return cudaSuccess;
    peak_array_kernel<<<grid_for(nSeries), kBlock, 0, st>>>(data, nSeries, len, h, cap, counts, peaks, intervals);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_point_dbscan(const double* intervals, const int* counts, long long n, int stride, double eps,
                                int* labScratch, int* slotScratch, int* out, cudaStream_t st, const int* outIdx) {
    if (n <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((n * 32 + kBlock - 1) / kBlock);
    const size_t shared = (size_t)(kBlock / 32) * std::min(stride, kDbscanBits) * sizeof(float);
    point_dbscan_kernel<false><<<grid, kBlock, shared, st>>>(intervals, counts, n, stride, eps, labScratch, slotScratch,
                                                             out, outIdx);
    note_launch();
    if (stride > kDbscanBits) {
        point_dbscan_kernel<true><<<grid, kBlock, 0, st>>>(intervals, counts, n, stride, eps, labScratch, slotScratch,
                                                           out, outIdx);
        note_launch();
    }
    return cudaGetLastError();
}

cudaError_t launch_trajectory_f64(int system, const double* x0, const double* a0, double h, int nSteps,
                                  double* out, long long n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
#define CALL(S) \
    (trajectory_kernel<S><<<grid_for(n), kBlock, 0, st>>>(x0, a0, h, nSteps, out, n), note_launch())
    CHAOS_SYSTEM_SWITCH(system, CALL)
#undef CALL
    return cudaGetLastError();
}

}  // namespace chaos
