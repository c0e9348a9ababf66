// FP64 sweeps of the RK4 systems with a team of three lanes per trajectory, one
// state component each: small sweeps, which leave schedulers idle.
//
// Why: on this GPU an FP64 warp instruction occupies its scheduler's share of
// the pipe for 64 cycles however many lanes are active, and a lone warp
// waits for every one of them. A sweep of up to a few thousand points has
// fewer warps than the GPU has schedulers (999 points: 32 of 608), so its
// time is the number of FP64 instructions of one warp. With a component per
// lane the three components of a stage are one instruction: a Lorenz step
// takes 15 instead of 45, for 10 points per warp instead of 32; the lanes
// exchange their stage values by shuffles and select the operands of their
// component's formula, on pipes that are idle here.
//
// Every component's value is rounded exactly as step() rounds it: a product
// is fma(a, b, -0), a difference of two values fma(1, a, -b) (or fma(-1, b,
// a)), each equal to the single operation, signed zeros included.
//
// Included by kern_f64.cu (compiled with --fmad=false).
#pragma once

#include "engine.cuh"

namespace chaos {

// Ten teams a warp; lanes 30 and 31 repeat lanes 0 and 1 (their results are
// not used, but they take part in the shuffles). s1 and s2 hold the
// components after this lane's in cyclic order.
struct TeamLane {
    static constexpr int kTeams = 10;
    int team, role, base, s1, s2;
    __device__ __forceinline__ TeamLane() {
        const int lane = threadIdx.x & 31, l = lane < 30 ? lane : lane - 30;
        team = l / 3;
        role = l % 3;
        base = 3 * team;
        s1 = base + (role + 1) % 3;
        s2 = base + (role + 2) % 3;
    }
    __device__ __forceinline__ bool spare() const { return (threadIdx.x & 31) >= 30; }
    static __device__ __forceinline__ double from(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
    // sqrt-free sum of squares of the team's values in component order, each operation rounded apart
    __device__ __forceinline__ double sum_squares(double d) const {
        const double q = d * d;
        return (from(q, base) + from(q, base + 1)) + from(q, base + 2);
    }
};

// -v on the integer pipe (the compiler's negation of a double that is not
// folded into an operation takes an FP64 instruction).
__device__ __forceinline__ double flip(double v) {
    return __hiloint2double(__double2hiint(v) ^ (int)0x80000000, __double2loint(v));
}

// own component's derivative from the own value x and the team's others,
// A = component role + 1, B = component role + 2 (cyclic).
template <class F> struct TeamField;

template <> struct TeamField<Lorenz> {
    bool r0, r1, r2;
    double p, c, u;  // {1, -1, beta}, {., rho, -0}, {sigma, ., .}
    __device__ __forceinline__ TeamField(const double* a, int role) : r0(role == 0), r1(role == 1), r2(role == 2) {
        p = r0 ? 1.0 : (r1 ? -1.0 : a[2]);
        c = r1 ? a[1] : -0.0;
        u = a[0];
    }
    __device__ __forceinline__ double operator()(double x, double A, double B) const {
        const double t = fma(p, r2 ? x : A, r0 ? flip(x) : c);  // y - x | rho - z | beta z
        // sigma t | x t - y | x y - t
        return fma(r0 ? u : (r1 ? B : A), r2 ? B : t, flip(r0 ? 0.0 : (r1 ? x : t)));
    }
};

template <> struct TeamField<Rossler> {
    bool r0, r1, r2;
    double c, u, w;  // {., ., -c}, {-1, a, .}, {-0, ., b}
    __device__ __forceinline__ TeamField(const double* a, int role) : r0(role == 0), r1(role == 1), r2(role == 2) {
        c = -a[2];
        u = r0 ? -1.0 : a[0];
        w = r0 ? -0.0 : a[1];
    }
    __device__ __forceinline__ double operator()(double x, double A, double B) const {
        const double t = A + (r0 ? B : c);  // y + z | . | x - c
        return fma(r2 ? x : u, r1 ? x : t, r1 ? B : w);  // -t | a y + x | z t + b
    }
};

template <> struct TeamField<Chen> {
    bool r0, r1, r2;
    double p, c, u, s;  // {1, -1, b}, {., c - a, -0}, {a, ., .}, c
    __device__ __forceinline__ TeamField(const double* a, int role) : r0(role == 0), r1(role == 1), r2(role == 2) {
        p = r0 ? 1.0 : (r1 ? -1.0 : a[1]);
        c = r1 ? a[2] - a[0] : -0.0;
        u = a[0];
        s = a[2];
    }
    __device__ __forceinline__ double operator()(double x, double A, double B) const {
        const double t = fma(p, r2 ? x : A, r0 ? flip(x) : c);  // y - x | (c - a) - z | b z
        const double cy = s * x;
        // a t | x t + c y | x y - t
        return fma(r0 ? u : (r1 ? B : A), r2 ? B : t, r1 ? cy : flip(r0 ? 0.0 : t));
    }
};

// One classic RK4 step of M trajectories (rk4_step's stages and sums), one
// component of each per lane; the M chains overlap.
template <int M, class F>
__device__ __forceinline__ void team_step(double* x, const TeamField<F>& f, const RK4H<double>& c, const TeamLane& l) {
    double k[M], y[M], acc[M];
#pragma unroll
    for (int m = 0; m < M; ++m) k[m] = f(x[m], l.from(x[m], l.s1), l.from(x[m], l.s2));
#pragma unroll
    for (int m = 0; m < M; ++m) {
        acc[m] = k[m];
        y[m] = fma(c.hh, k[m], x[m]);
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) {
#pragma unroll
        for (int m = 0; m < M; ++m) k[m] = f(y[m], l.from(y[m], l.s1), l.from(y[m], l.s2));
        if (s < 2) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                y[m] = fma(s == 0 ? c.hh : c.h, k[m], x[m]);
                acc[m] = fma(2.0, k[m], acc[m]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) x[m] = fma(c.h6, addR(acc[m], k[m]), x[m]);
}

__device__ __forceinline__ double of_role(const double* v, int role) {
    return role == 0 ? v[0] : (role == 1 ? v[1] : v[2]);
}

// v > p for finite values on the integer pipe (an FP64 compare would take an
// FP64 instruction's 64 cycles): order keys, the two zeros alike.
__device__ __forceinline__ bool above(double v, double p) {
    auto key = [](double d) {
        const long long b = __double_as_longlong(d);
        return b >= 0 ? b : (long long)0x8000000000000000ull - b;
    };
    return key(v) > key(p);
}

// The recorded loop of a warp's teams: B samples, one before each advance of
// the warp. The lane that holds the recorded component (rec on entry: a point
// in use that records) keeps the samples, judges them in windows and tests
// for divergence, as record_windows does; it returns 0 when the point
// diverged and 1 otherwise, rec false after a divergence, xp (every lane) the
// value before the last advance, last the last sample.
constexpr int kTeamWindow = 32;
constexpr int kTeamColumn = kTeamWindow + 3;  // doubles per team: odd, so that the teams' stores spread over the banks

template <class Advance, class Diverged, class OnPeak>
__device__ __forceinline__ int team_record(int B, double& x, double& xp, double* col, bool& rec, PeakWindow& d,
                                           double& last, Advance&& advance, Diverged&& diverged, OnPeak&& on_peak) {
    constexpr int K = kTeamWindow;
    auto at = [&](int j) { return col[j + 2]; };
    auto judge = [&](int k, unsigned mask, unsigned up, int m) {
        unsigned cand = PeakWindow::candidates(mask, up, m);
        auto peak = [&](double val, int t) {
            on_peak(val, t);
            d.tprev = t;
            ++d.n;
        };
        // (a plateau whose window is all one value goes on)
        if (d.i0 >= 0 && (mask != 0u || at(m - 1) != at(-1))) d.walk(k, 0, m, at, peak);
        while (cand != 0u) {
            const int j = PeakWindow::next(cand, m);
            d.judge(k, j, m, at, peak);
        }
    };
    d.init();
    int flag = 1;
    unsigned up = 0;
    double p = 0.0;
    if (rec) col[0] = col[1] = 0.0;
    xp = x;
    // The first window is one sample: it ends the points that were beyond the
    // bound before they were recorded, where a window would be most of their time
    // (150^2 Lorenz points, all of them beyond, 5 steps a sample, 0.34 -> 0.04 ms).
    for (int i = 0, most = 1, m; i < B; i += m, most = K) {
        m = min(most, B - i);
        unsigned mask = 0;
        int bad = K + 1;  // samples before the divergent one, when there is one
#pragma unroll 2
        for (int j = 0; j < m; ++j) {
            xp = x;
            mask = (mask << 1) | (above(x, p) ? 1u : 0u);
            p = x;
            if (rec) col[j + 2] = x;
            advance();
            if (diverged(x)) bad = min(bad, j + 1);
        }
        if (rec) {
            if (bad <= m) {
                judge(i, mask >> (m - bad), up, bad);
                last = col[bad + 1];
                rec = false;
                flag = 0;
            } else {
                judge(i, mask, up, m);
                last = p;
                col[0] = col[m];
                col[1] = p;
            }
        }
        up = mask & 1u;
        if (!__any_sync(0xffffffffu, rec)) break;
    }
    return flag;
}

// Bifurcation points (bif_point), ten per warp.
template <class F>
__device__ __forceinline__ void bif_teams(const SweepParams& P, const BifOut& O, double* cols) {
    const TeamLane l;
    long long o = (long long)blockIdx.x * TeamLane::kTeams + l.team;
    const bool used = !l.spare() && o < P.nPoints;
    if (o >= P.nPoints) o = P.nPoints - 1;
    double xs[3], as[3];
    load_point<SYS_LORENZ_RK4, double>(P, P.pBegin + o, xs, as);  // any 3-state, 3-parameter system loads alike
    const TeamField<F> f(as, l.role);
    const RK4H<double> c(P.h);
    double x = of_role(xs, l.role), xp = x;
    const bool owner = used && l.role == P.wv;  // the lane that watches and records
    bool live = owner;
    if (P.S > 0) {
        int s = 0;
        bool any = true;  // some point of the warp has not diverged
        for (; s + kTransientBlock <= P.S - 1 && any; s += kTransientBlock) {
            bool dv = false;
#pragma unroll
            for (int j = 0; j < kTransientBlock; ++j) {
                team_step<1>(&x, f, c, l);
                dv |= bif_diverged(x, P);
            }
            if (dv) live = false;
            any = __any_sync(0xffffffffu, live);
        }
        for (; s < P.S && any; ++s) {
            xp = x;
            team_step<1>(&x, f, c, l);
            if (bif_diverged(x, P)) live = false;
        }
        const double d = x - xp;
        if ((double)sqrtf(fabsf((float)l.sum_squares(d))) < 1e-9) live = false;  // fixed: reported as diverged
    }
    const double first = live ? x : 0.0;
    double* pk = O.peaks ? O.peaks + o * (long long)O.cap : nullptr;
    double* iv = O.intervals ? O.intervals + o * (long long)O.cap : nullptr;
    bool rec = live;
    PeakWindow d;
    d.init();
    double last;
    int flag = 0;
    if (__any_sync(0xffffffffu, live)) {
        flag = team_record(
            P.B, x, xp, cols + kTeamColumn * l.team, rec, d, last, [&] { team_step<1>(&x, f, c, l); },
            [&](double v) { return bif_diverged(v, P); },
            [&](double val, int t) {
                const int q = d.n - 1;
                if (q >= 0 && q < O.cap) {
                    if (pk) pk[q] = val;
                    if (iv) iv[q] = __dmul_rn((double)(t - d.tprev), P.hInterval);
                }
            });
        const double dx = x - xp;
        if ((double)sqrtf(fabsf((float)l.sum_squares(dx))) < 1e-9 && flag == 1) flag = -1;
    }
    if (!owner) return;
    if (!live) flag = 0;
    const int kept = d.n > 1 ? d.n - 1 : 0;
    O.flags[o] = flag;
    O.counts[o] = flag == 1 ? kept : (flag == -1 ? -1 : 0);
    if (O.first) O.first[o] = first;
}

// Basins points (basins_point), ten per warp.
template <class F>
__device__ __forceinline__ void basins_teams(const SweepParams& P, const BasinsOut& O, double* cols) {
    const TeamLane l;
    long long o = (long long)blockIdx.x * TeamLane::kTeams + l.team;
    const bool used = !l.spare() && o < P.nPoints;
    if (o >= P.nPoints) o = P.nPoints - 1;
    double xs[3], as[3];
    load_point<SYS_LORENZ_RK4, double>(P, P.pBegin + o, xs, as);
    const TeamField<F> f(as, l.role);
    const RK4H<double> c(P.h);
    double x = of_role(xs, l.role), xp;
#pragma unroll 4
    for (int s = 0; s < P.S; ++s) team_step<1>(&x, f, c, l);
    const bool owner = used && l.role == P.wv;
    bool rec = owner;
    PeakWindow d;
    PeakSums<double> sums;
    double last = 0.0;
    int flag = team_record(
        P.B, x, xp, cols + kTeamColumn * l.team, rec, d, last,
        [&] {
#pragma unroll 1
            for (int r = 0; r < P.preScaller; ++r) team_step<1>(&x, f, c, l);
        },
        [&](double v) { return basins_diverged(v, P); },
        [&](double val, int t) {
            if (d.n >= 1) sums.add(val, t - d.tprev, P.hInterval);
        });
    const double dx = x - xp;
    if (sqrt(fabs(l.sum_squares(dx))) < 1e-9 && flag == 1) flag = -1;
    if (!owner) return;
    write_basins_point(O, o, flag, d.n > 1 ? d.n - 1 : 0, sums.peaks(), sums.intervals(P.hInterval), last);
}

// LLE points (lle_point_full): the orbit and its twin, both in the lanes of
// one team (G = 1, ten points a warp) or in a team each (G = 2: lanes 0..14
// the orbits of five points, 15..29 their twins; half the instructions a
// step, for sweeps that still leave schedulers idle then).
template <class F, int G>
__device__ __forceinline__ void lle_teams(const LleParams& L, double* out) {
    constexpr int kPoints = TeamLane::kTeams / G, M = 2 / G;
    const TeamLane l;
    const bool twin = G == 2 && l.team >= kPoints;  // this lane's trajectory is the twin
    long long o = (long long)blockIdx.x * kPoints + l.team % kPoints;
    const bool writes = !l.spare() && l.role == 0 && !twin && o < L.nPoints;
    if (o >= L.nPoints) o = L.nPoints - 1;
    double xs[3], as[3];
    lle_load<3, 3>(L, L.pBegin + o, xs, as);
    const TeamField<F> f(as, l.role);
    const RK4H<double> c(L.h);
    double v[2];  // the orbit's component and the twin's, or (G = 2) the own trajectory's
    v[0] = of_role(xs, l.role);
#pragma unroll 4
    for (int s = 0; s < L.trans; ++s) team_step<1>(v, f, c, l);  // (G = 2: the twins' lanes run the same orbit)
    double q = v[0];
    if (L.twin == 1) q = (double)__fmaf_rn(l.role == 0 ? 1.0f : 0.0f, (float)L.eps, (float)v[0]);
    else if (l.role == 0) q = v[0] + L.eps;
    if (G == 1) v[1] = q;
    else if (twin) v[0] = q;
    const int partner = (threadIdx.x & 31) < 30 ? (l.base + l.role + 15) % 30 : 15 + l.role;
    double sum = 0.0;
    for (int b = 0; b <= L.calcBlocks; ++b) {
#pragma unroll 2
        for (int s = 0; s < L.ntp; ++s) team_step<M>(v, f, c, l);
        double x, y;  // this component of the orbit and of the twin
        if (G == 1) {
            x = v[0];
            y = v[1];
        } else {
            const double other = l.from(v[0], partner);
            x = twin ? other : v[0];
            y = twin ? v[0] : other;
        }
        const double df = x - y;
        const double dist = sqrt(l.sum_squares(df)) / L.eps;
        sum = sum + log(dist);
        y = x - df / dist;
        if (G == 1) v[1] = y;
        else if (twin) v[0] = y;
    }
    if (writes) out[o] = sum / L.tMax;
}

// Spectrum points (spectrum_point_full): the orbit and its three twins, all in
// the lanes of one team (G = 1, ten points a warp) or in a team each (G = 4, two
// points a warp, teams 8 and 9 idle along). Between blocks every lane holds its
// component of all four, the dot products are sums over the team's lanes in
// component order, and with G = 4 a team takes its own twin's norm and logarithm.
template <class F, int G>
__device__ __forceinline__ void spectrum_teams(const LleParams& L, double* out) {
    constexpr int kPoints = G == 1 ? TeamLane::kTeams : 2, M = 4 / G;
    const TeamLane l;
    const int point = G == 1 ? l.team : min(l.team / 4, 1);
    const int traj = G == 1 ? 0 : l.team % 4;  // of this lane: 0 the orbit
    long long o = (long long)blockIdx.x * kPoints + point;
    const bool writes = !l.spare() && l.role == 0 && o < L.nPoints && (G == 1 || (traj > 0 && l.team < 8));
    if (o >= L.nPoints) o = L.nPoints - 1;
    double xs[3], as[3];
    lle_load<3, 3>(L, L.pBegin + o, xs, as);
    const TeamField<F> f(as, l.role);
    const RK4H<double> c(L.h);
    double v[M], sum[3] = {0.0, 0.0, 0.0};  // (G = 4: its own twin's in sum[0])
    v[0] = of_role(xs, l.role);
#pragma unroll 4
    for (int s = 0; s < L.trans; ++s) team_step<1>(v, f, c, l);
    if (G == 1) {
#pragma unroll
        for (int j = 1; j < M; ++j) v[j] = l.role == j - 1 ? v[0] + L.eps : v[0];
    } else if (l.role == traj - 1) {
        v[0] = v[0] + L.eps;
    }
    // sum of the team's products in component order from 0.0: a sum of -0 is +0
    auto dot = [&](double a, double b) {
        const double q = a * b, t = (l.from(q, l.base) + l.from(q, l.base + 1)) + l.from(q, l.base + 2);
        return __double2hiint(t) == (int)0x80000000 && __double2loint(t) == 0 ? 0.0 : t;
    };
    for (int b = 0; b <= L.calcBlocks; ++b) {
#pragma unroll 2
        for (int s = 0; s < L.ntp; ++s) team_step<M>(v, f, c, l);
        double x = v[0], d[3], g[3];
        if (G == 1) {
#pragma unroll
            for (int j = 0; j < 3; ++j) d[j] = v[(j + 1) % M] - x;
        } else {
            x = l.from(v[0], 12 * point + l.role);
#pragma unroll
            for (int j = 0; j < 3; ++j) d[j] = l.from(v[0], 12 * point + 3 * (j + 1) + l.role) - x;
        }
        double den[2];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            g[j] = d[j];
#pragma unroll
            for (int m = 0; m < j; ++m) {
                const double num = dot(d[j], g[m]);
                const double frac = den[m] == 0.0 ? 0.0 : num / den[m];
                g[j] = g[j] - frac * g[m];
            }
            if (j < 2) den[j] = l.sum_squares(g[j]);
        }
        auto renorm = [&](double gj, double& s) {
            const double nrm = sqrt(l.sum_squares(gj));
            s = s + log(nrm / L.eps);
            return x + (nrm == 0.0 ? 0.0 : gj / nrm) * L.eps;
        };
        if (G == 1) {
#pragma unroll
            for (int j = 0; j < 3; ++j) v[(j + 1) % M] = renorm(g[j], sum[j]);
        } else {
            const double y = renorm(of_role(g, max(traj - 1, 0)), sum[0]);
            if (traj > 0) v[0] = y;
        }
    }
    if (!writes) return;
    double* row = out + (L.pBegin + o) * 3;
    if (G == 1) {
#pragma unroll
        for (int j = 0; j < 3; ++j) row[j] = sum[j] / L.tMax;
    } else {
        row[traj - 1] = sum[0] / L.tMax;
    }
}

}  // namespace chaos
