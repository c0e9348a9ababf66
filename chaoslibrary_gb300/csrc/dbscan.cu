// Grid clustering on the device, cell first.
//
// Both clusterings (textbook DBSCAN and the reference's eps-components) run
// one pipeline over points in a D-dimensional feature space (D = 1..3). The
// points are read from a feature source: feature columns, a row-major matrix,
// or the basin map's per-point outputs normalised on the fly. The work is
// arranged so that a map's millions of points are read once and touched
// again only through 4-byte cell slots, while exact point tests run on the
// few cells that need them:
//   1. one pass over the points: the cell of every point (floor(f / side) per
//      dimension, side = eps / sqrt(D) shrunk by 1e-9, so two points of one
//      cell are always within eps and a neighbour within eps is at most R = 2
//      cells away per dimension) goes into an open-addressing hash table with
//      the cell's point count, bounding box (float bounds rounded outward:
//      still a box around the points), smallest index and another one (its
//      representatives), smallest fixed-point index and a clamped/NaN mark,
//      gathered per block in shared memory; the point keeps its slot;
//   2. per cell: dense (a safe cell with >= minPts points -- every included
//      point in the reference mode: all its points are core) or not; the
//      occupied neighbour cells; per neighbouring pair, the bounding boxes
//      settle most pairs (farther than eps: nothing; every point within eps:
//      joined), the representatives join most other pairs of dense cells;
//      the joined pairs' components come from one block's union-find in
//      shared memory;
//   3. the points of the cells that are not dense are sorted by cell (one
//      pass over the slots) and their core flags counted: whole cells by
//      their boxes, dense cells' representatives as a lower bound, sorted
//      cells exactly; core points join dense neighbours the same way;
//   4. the cells that some pair, core count or border label still has to
//      scan -- pairs of dense cells that the unions so far leave apart, dense
//      neighbours of points whose count or label the shortcuts cannot settle
//      -- are sorted in a second pass, and their point pairs tested exactly;
//   5. union-find over nodes: a safe cell's core points are one node (they
//      are within eps of each other), a core point of a clamped/NaN cell is
//      a node of its own; lock-free hooking with atomicCAS, parent[v] <= v;
//   6. components numbered by their smallest core index (and, in the
//      reference mode, their smallest fixed-point index); one pass over the
//      slots writes the labels of the dense cells' points, a kernel over the
//      sorted points those of the others (border points: the component of
//      the smallest index among the core points within eps).
// Distances are sqrt(sum of squared differences) <= eps in FP64, in dimension
// order, each operation rounded on its own (this file is compiled with
// --fmad=false), as the reference computes them (Basins/src/basinsCUDA.cu:918);
// the square root is skipped where the squared distance is clear of eps^2 by
// 1e-7. Cells whose coordinates had to be clamped (|f| / side >= 2^19) or that
// hold a NaN feature lose the one-cell-is-connected shortcut and are resolved
// by exact pair tests. Every box test keeps a relative margin of 1e-7 on
// squared distances, and a representative is a real point of its cell, so the
// shortcuts skip work without changing a label.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "dbscan.h"
#include "order_keys.h"

namespace chaos {

namespace {

constexpr int kTPB = 256;
constexpr unsigned long long kEmpty = ~0ull;
constexpr long long kLim = 1LL << 19;  // clamp of cell coordinates (21-bit packing for D = 3)
constexpr int kR = 2;                  // neighbour reach in cells
constexpr int kReps = 2;               // representatives per cell: its smallest point index and another

__device__ __forceinline__ unsigned long long pack(const long long* c, int D) {
    if (D <= 2) {
        const unsigned long long a = (unsigned long long)(c[0] + 2147483648LL);
        const unsigned long long b = (unsigned long long)((D == 2 ? c[1] : 0) + 2147483648LL);
        return (a << 32) | (b & 0xffffffffull);
    }
    return (((unsigned long long)c[0] & 0x1FFFFFull) << 42) | (((unsigned long long)c[1] & 0x1FFFFFull) << 21) |
           ((unsigned long long)c[2] & 0x1FFFFFull);
}

__device__ __forceinline__ void unpack(unsigned long long k, int D, long long* c) {
    if (D <= 2) {
        c[0] = (long long)(k >> 32) - 2147483648LL;
        c[1] = (long long)(k & 0xffffffffull) - 2147483648LL;
        c[2] = 0;
        return;
    }
    for (int d = 0; d < 3; ++d) {
        long long v = (long long)((k >> (42 - 21 * d)) & 0x1FFFFFull);
        if (v & 0x100000) v -= 0x200000;
        c[d] = v;
    }
}

__device__ __forceinline__ unsigned long long mix(unsigned long long k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return k;
}

__device__ __forceinline__ double dist2(const double* a, const double* b, int D) {
    double s = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d >= D) continue;
        const double df = a[d] - b[d];
        s = s + df * df;
    }
    return s;
}

// ---- prefix sum ------------------------------------------------------------
constexpr int kScanItems = 4096;  // 1024 threads x 4

template <class T>
__global__ void __launch_bounds__(1024) scan_block_kernel(const T* in, T* out, T* blockSums, long long n) {
    __shared__ T warpSums[32];
    const long long base = (long long)blockIdx.x * kScanItems + threadIdx.x * 4;
    T v[4], s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        v[j] = base + j < n ? in[base + j] : 0;
        s += v[j];
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warpSums[w] = x;
    __syncthreads();
    if (w == 0) {
        T ws = warpSums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, ws, o);
            if (lane >= o) ws += y;
        }
        warpSums[lane] = ws;
    }
    __syncthreads();
    T prefix = (w > 0 ? warpSums[w - 1] : 0) + x - s;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (base + j < n) out[base + j] = prefix;
        prefix += v[j];
    }
    if (threadIdx.x == 1023) blockSums[blockIdx.x] = warpSums[31];
}

template <class T>
__global__ void add_offsets_kernel(T* out, const T* offsets, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += offsets[i / kScanItems];
}

inline unsigned blocks(long long n, int tpb = kTPB) { return (unsigned)((n + tpb - 1) / tpb); }

// ---- order keys (order_keys.h: okey, unkey, group_min64, group_max64) ------------
// Order keys of floats: the cell boxes are kept in float, each bound rounded
// outward (minima down, maxima up), so a box still holds all its points and
// every box test stays one-sided; 32-bit keys take the native atomics.
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unfkey(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
constexpr unsigned kFKeyPosInf = 0xff800000u;  // fkey(+inf)
constexpr unsigned kFKeyNegInf = 0x007fffffu;  // fkey(-inf)

// ---- cell boxes ------------------------------------------------------------------
// A cell's box holds all its points, so a box farther than eps from a point
// (or from another box) holds no point within eps, and a box whose farthest
// corner is within eps holds only points within eps. Both tests keep a
// relative margin of 1e-7 on the squared distance (far above the rounding of
// the exact test), so they never change a result, only skip work.
constexpr double kBoxOut = 1.0000001, kBoxIn = 0.9999999;

// sqrt(d2) <= eps, the reference's test, with the square root taken only near
// the boundary: a squared distance below eps^2 (1 - 1e-7) has its root below
// eps and one above eps^2 (1 + 1e-7) above it, far outside the roundings of
// the square, the product and the root; NaN is never within.
__device__ __forceinline__ bool within_eps(double d2, double eps) {
    const double eps2 = eps * eps;
    if (d2 <= eps2 * kBoxIn) return true;
    if (d2 > eps2 * kBoxOut) return false;
    return sqrt(d2) <= eps;
}

__device__ __forceinline__ void box_dist2(const double* v, const double* lo, const double* hi, int D, double& near2,
                                          double& far2) {
    near2 = 0.0;
    far2 = 0.0;
    for (int d = 0; d < D; ++d) {
        double g = 0.0;
        if (v[d] < lo[d]) g = lo[d] - v[d];
        else if (v[d] > hi[d]) g = v[d] - hi[d];
        near2 = near2 + g * g;
        const double f = fmax(fabs(v[d] - lo[d]), fabs(hi[d] - v[d]));
        far2 = far2 + f * f;
    }
}

// ---- counts the pipeline keeps on the device ---------------------------------------
// The sizes of the later steps stay in device memory: their kernels read them
// (a fixed grid loops over the work). The host waits for the number of cells,
// and in large sets for a bound on it, for the neighbour entries and for the
// sorted points (cell_cluster).
enum Count {
    kCells, kErr, kEntries, kOpen, kJoinedCount, kSparse, kNeeded, kActive, kLong, kScanA, kScanB, kCounts
};
constexpr int kLoopBlocksPerSm = 8;  // blocks of kTPB threads of a looping kernel

__device__ __forceinline__ long long first_warp() { return ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
__device__ __forceinline__ long long warp_stride() { return ((long long)gridDim.x * blockDim.x) >> 5; }
// sorted points, and nodes of the union-find over cells and sorted points
__device__ __forceinline__ int sorted_points(const int* counts) { return counts[kSparse] + counts[kNeeded]; }

// ---- union-find (parent[v] <= v) --------------------------------------------
__device__ __forceinline__ int uf_find(int* parent, int x) {
    int cur = __ldcg(parent + x);
    if (cur != x) {
        int prev = x, next;
        while (cur > (next = __ldcg(parent + cur))) {
            parent[prev] = next;
            prev = cur;
            cur = next;
        }
    }
    return cur;
}

__device__ __forceinline__ void uf_unite(int* parent, int a, int b) {
    int ra = uf_find(parent, a), rb = uf_find(parent, b);
    while (ra != rb) {
        if (ra < rb) { const int t = ra; ra = rb; rb = t; }
        const int old = atomicCAS(parent + ra, ra, rb);
        if (old == ra) break;
        ra = old;
        rb = uf_find(parent, rb);
        ra = uf_find(parent, ra);
    }
}

// warp-aggregated append of p to list (one atomic per warp)
__device__ __forceinline__ void list_append(bool take, int p, int* list, int* count) {
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (!m) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (take) list[base + __popc(m & ((1u << lane) - 1))] = p;
}

// ---- feature sources ---------------------------------------------------------
// Where the clustering reads point i: whether it takes part, its features
// (FP64) and, for the reference-compatible numbering, whether it is a fixed
// point (flag -1).
struct ColSrc {  // feature columns
    const double* f[3];
    const int* mask;   // textbook mode: the points with mask[i] != 0 (all when null)
    const int* flags;  // reference mode: the points with flags[i] != 0
    int D;
    bool compat;
    __device__ __forceinline__ bool included(long long i) const {
        return compat ? flags[i] != 0 : (mask ? mask[i] != 0 : true);
    }
    __device__ __forceinline__ bool fix(long long i) const { return compat && flags[i] == -1; }
    __device__ __forceinline__ void load(long long i, double* v) const {
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (d < D) v[d] = f[d][i];
    }
};

struct RowSrc {  // row-major n x D matrix, textbook mode
    const double* F;
    const int* mask;
    int D;
    __device__ __forceinline__ bool included(long long i) const { return mask ? mask[i] != 0 : true; }
    __device__ __forceinline__ bool fix(long long) const { return false; }
    __device__ __forceinline__ void load(long long i, double* v) const {
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (d < D) v[d] = F[i * D + d];
    }
};

// The basin map's outputs, normalised on the fly: per point (amplitude, kept
// peak count, mean interval) -- the amplitude is the mean peak value, or the
// last recorded sample for a point without peaks -- min-max scaled per
// feature over the points with flag != 0: (f - lo) * (1 / (hi - lo)), 0 for a
// feature whose points are all equal.
struct BasinSrc {
    const int* flags;
    const int* counts;
    const double* avgPeaks;
    const double* avgIntervals;
    const double* last;
    double lo[3], inv[3];
    int ok[3];
    int D;
    __device__ __forceinline__ bool included(long long i) const { return flags[i] != 0; }
    __device__ __forceinline__ bool fix(long long) const { return false; }
    __device__ __forceinline__ void load(long long i, double* v) const {
        const int c = counts[i];
        const double f[3] = {c > 0 ? avgPeaks[i] : last[i], (double)c, c > 0 ? avgIntervals[i] : 0.0};
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = ok[d] ? (f[d] - lo[d]) * inv[d] : 0.0;
    }
};

// ---- the cell table: slot-indexed statistics of the occupied cells ---------------
struct alignas(16) CellStats {
    unsigned lo[3];  // order keys of the feature minima rounded down to float
    unsigned hi[3];  // order keys of the feature maxima rounded up to float
    int cnt;         // points
    int bad;         // a clamped or NaN point
    int minIdx;      // smallest point index
    int other;       // some point's index, mostly far from the smallest (-1: none yet)
    int minFix;      // smallest fixed-point index (reference mode)
    int pad;
};
struct Table {
    unsigned long long* key;  // packed cell coordinates, kEmpty for a free slot
    unsigned long long mask;  // capacity - 1 (a power of two)
    CellStats* st;
};

__device__ __forceinline__ CellStats empty_stats() {
    CellStats s;
    for (int d = 0; d < 3; ++d) {
        s.lo[d] = kFKeyPosInf;
        s.hi[d] = kFKeyNegInf;
    }
    s.cnt = 0;
    s.bad = 0;
    s.minIdx = INT_MAX;
    s.other = -1;
    s.minFix = INT_MAX;
    s.pad = 0;
    return s;
}

__global__ void table_init_kernel(Table T, long long cap) {
    const long long h = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= cap) return;
    T.key[h] = kEmpty;
    T.st[h] = empty_stats();
}

__device__ __forceinline__ long long table_insert(unsigned long long* tab, unsigned long long mask,
                                                  unsigned long long k) {
    unsigned long long g = mix(k) & mask;
    for (unsigned long long probe = 0; probe <= mask; ++probe) {
        const unsigned long long prev = atomicCAS(&tab[g], kEmpty, k);
        if (prev == kEmpty || prev == k) return (long long)g;
        g = (g + 1) & mask;
    }
    return -1;  // only if the table were full (it has twice as many slots as cells)
}

__device__ __forceinline__ int hash_find(const unsigned long long* tab, unsigned long long mask, const int* slotCell,
                                         unsigned long long k) {
    unsigned long long h = mix(k) & mask;
    for (unsigned long long probe = 0; probe <= mask; ++probe) {
        const unsigned long long t = tab[h];
        if (t == k) return slotCell[h];
        if (t == kEmpty) return -1;
        h = (h + 1) & mask;
    }
    return -1;
}

// NaN test on the bits (the integer pipe; a double compare takes the FP64 pipe)
__device__ __forceinline__ bool is_nan(double v) {
    return ((unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull;
}

// Cell coordinates of a feature vector; true when the point is clamped or NaN.
// q = f * (1/side): the rounding of the product (|q| < 2^19: below 1e-10 of a
// cell) stays far inside the 1e-9 by which the side is shrunk, so two points
// of one cell are still within eps. floor(q) is one conversion rounding down
// (saturating for infinities), clamped on the integer.
__device__ __forceinline__ bool cell_coords(const double* v, int D, double invSide, long long* c) {
    bool bad = false, nan = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d >= D) continue;
        const double q = v[d] * invSide;
        nan = nan || is_nan(q);
        long long k = __double2ll_rd(q);
        if (k >= kLim) { k = kLim; bad = true; }
        else if (k < -kLim) { k = -kLim; bad = true; }
        c[d] = k;
    }
    if (nan) {
        c[0] = c[1] = c[2] = kLim + 5;
        return true;
    }
    return bad;
}

// Extent of the cell coordinates of the ordinary points (ext[d] = -min,
// ext[3 + d] = max) and the number of clamped or NaN ones (ext[6]): the
// occupied cells are at most the product of the extents plus that count,
// which sizes the table. Warps reduce with shuffles into shared memory, one
// global atomic per block and quantity. (Sources whose features have known
// bounds skip this pass.)
template <class Src>
__global__ void extent_kernel(Src S, long long n, double invSide, long long* ext) {
    __shared__ long long sext[7];
    if (threadIdx.x < 7) sext[threadIdx.x] = threadIdx.x < 6 ? LLONG_MIN : 0;
    __syncthreads();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long c[3] = {0, 0, 0};
    bool bad = false, ok = false;
    if (i < n && S.included(i)) {
        double v[3];
        S.load(i, v);
        bad = cell_coords(v, S.D, invSide, c);
        ok = !bad;
    }
    const int lane = threadIdx.x & 31;
    const unsigned nbad = __popc(__ballot_sync(0xffffffffu, bad));
    if (lane == 0 && nbad) atomicAdd((unsigned long long*)&sext[6], (unsigned long long)nbad);
    if (__any_sync(0xffffffffu, ok)) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (d >= S.D) continue;
            long long lo = ok ? -c[d] : LLONG_MIN, hi = ok ? c[d] : LLONG_MIN;  // max of -c and of c
            for (int o = 16; o > 0; o >>= 1) {
                lo = max(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            if (lane == 0) {
                atomicMax(&sext[d], lo);
                atomicMax(&sext[3 + d], hi);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 6 && sext[threadIdx.x] != LLONG_MIN) atomicMax(&ext[threadIdx.x], sext[threadIdx.x]);
    if (threadIdx.x == 6 && sext[6]) atomicAdd((unsigned long long*)&ext[6], (unsigned long long)sext[6]);
}

// The slot of a cell key: found by reading the table (no atomics once the
// cell is in it), inserted with atomicCAS otherwise.
__device__ __forceinline__ long long table_slot(unsigned long long* tab, unsigned long long mask,
                                                unsigned long long k) {
    unsigned long long g = mix(k) & mask;
    for (unsigned long long probe = 0; probe <= mask; ++probe) {
        const unsigned long long t = __ldcg(tab + g);
        if (t == k) return (long long)g;
        if (t == kEmpty) return table_insert(tab, mask, k);  // from here on, with atomics
        g = (g + 1) & mask;
    }
    return -1;
}

// Step 1. Each block takes a contiguous run of points and folds them into a
// small table of cells in shared memory, which it adds to the cell table at
// its end: the lanes of a warp that share a cell form a group, whose first
// lane finds (or claims) the cell's entry, adds the group's count and keeps
// its smallest and largest index; a lane whose point lies outside the box it
// reads widens it. A group that finds no room goes to the cell table itself.
// Bound by the FP64 pipe, which takes the points to their cells (81 % busy; 8
// million points in 3-D 0.31 ms, 0.68 TB/s). Folding every run of equal cells straight
// into the cell table, with an atomic per quantity, spent its time on the
// addresses of the few cells that hold most points: 1,000,000 points in
// random order 480 -> 55 us, a 2048^2 basin map 284 -> 273 us; reading a cell's
// values there before an atomic (1,440 us) waits at the same addresses.
constexpr int kCellBlock = 512, kCellBlocksPerSm = 2;
constexpr int kBlockCells = 512;  // entries of a block's table, a power of two
constexpr int kBlockProbes = 4;

struct BlockCells {
    unsigned long long key[kBlockCells];
    int slot[kBlockCells];  // in the cell table, -1 until found
    CellStats st[kBlockCells];
};

// Adds a cell's statistics (of some of its points) to its slot.
__device__ __forceinline__ void fold_stats(CellStats* to, const CellStats& s, int D, long long n) {
    atomicAdd(&to->cnt, s.cnt);
    if (s.minIdx < __ldcg(&to->minIdx)) atomicMin(&to->minIdx, s.minIdx);
    const int other = __ldcg(&to->other);
    if (other < 0 || s.other - other > (int)(n >> 6)) __stcg(&to->other, s.other);  // (any writer's will do)
    if (s.minFix != INT_MAX) atomicMin(&to->minFix, s.minFix);
    if (s.bad) atomicOr(&to->bad, 1);
    for (int d = 0; d < D; ++d) {
        if (s.lo[d] < __ldcg(&to->lo[d])) atomicMin(&to->lo[d], s.lo[d]);
        if (s.hi[d] > __ldcg(&to->hi[d])) atomicMax(&to->hi[d], s.hi[d]);
    }
}

// Fout (basin maps, when the caller asks for the normalised features) receives
// each point's row. chunk: points of a block, a multiple of its threads.
template <class Src>
__global__ void __launch_bounds__(kCellBlock, kCellBlocksPerSm)
cells_kernel(Src S, long long n, long long chunk, double invSide, Table T, int* slot, double* Fout, int* err) {
    extern __shared__ unsigned long long cell_smem[];
    BlockCells& B = *reinterpret_cast<BlockCells*>(cell_smem);
    for (int e = threadIdx.x; e < kBlockCells; e += blockDim.x) {
        B.key[e] = kEmpty;
        B.slot[e] = -1;
        B.st[e] = empty_stats();
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long begin = blockIdx.x * chunk, end = begin + chunk < n ? begin + chunk : n;
    for (long long i0 = begin; i0 < end; i0 += blockDim.x) {
        const long long i = i0 + threadIdx.x;
        unsigned long long key = kEmpty;
        double v[3] = {0.0, 0.0, 0.0};
        bool bad = false, fix = false;
        if (i < end && S.included(i)) {
            S.load(i, v);
            long long c[3] = {0, 0, 0};
            bad = cell_coords(v, S.D, invSide, c);
            key = pack(c, S.D);
            fix = S.fix(i);
        }
        if (Fout && i < end)
            for (int d = 0; d < 3; ++d) Fout[i * 3 + d] = v[d];
        // the lanes of this lane's cell (a row of one cell, common in a map, without the match)
        const unsigned long long key0 = __shfl_sync(0xffffffffu, key, 0);
        const unsigned grp = __all_sync(0xffffffffu, key == key0) ? 0xffffffffu : __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(grp) - 1;
        int e = -1, h = -1;  // the entry of the block's table (-1: no room), the slot of the cell table
        if (lane == leader && key != kEmpty) {
            unsigned p = (unsigned)(mix(key) >> 40);
            for (int k = 0; k < kBlockProbes; ++k, ++p) {
                const int q = (int)(p & (kBlockCells - 1));
                unsigned long long t = *(volatile unsigned long long*)&B.key[q];
                if (t == kEmpty) {
                    t = atomicCAS(&B.key[q], kEmpty, key);
                    if (t == kEmpty) t = key;
                }
                if (t == key) {
                    e = q;
                    h = *(volatile int*)&B.slot[q];
                    break;
                }
            }
            if (h < 0) {
                h = (int)table_slot(T.key, T.mask, key);
                if (h < 0) atomicAdd(err, 1);
                if (e >= 0) *(volatile int*)&B.slot[e] = h;
            }
        }
        e = __shfl_sync(0xffffffffu, e, leader);
        h = __shfl_sync(0xffffffffu, h, leader);
        if (i < end) slot[i] = key == kEmpty ? -1 : h;
        const unsigned fixes = __ballot_sync(0xffffffffu, fix) & grp;
        const unsigned bads = __ballot_sync(0xffffffffu, bad) & grp;
        if (key == kEmpty || h < 0) continue;
        unsigned lo[3], hi[3];  // the point's box (float, rounded outward)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const bool skip = d >= S.D || is_nan(v[d]);
            lo[d] = skip ? kFKeyPosInf : fkey(__double2float_rd(v[d]));
            hi[d] = skip ? kFKeyNegInf : fkey(__double2float_ru(v[d]));
        }
        const int last = (int)(i - lane) + 31 - __clz(grp);
        const int firstFix = fixes ? (int)(i - lane) + __ffs(fixes) - 1 : INT_MAX;
        if (e >= 0) {
            CellStats& st = B.st[e];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (d >= S.D) continue;
                if (lo[d] < *(volatile unsigned*)&st.lo[d]) atomicMin(&st.lo[d], lo[d]);
                if (hi[d] > *(volatile unsigned*)&st.hi[d]) atomicMax(&st.hi[d], hi[d]);
            }
            if (lane == leader) {
                atomicAdd(&st.cnt, __popc(grp));
                atomicMin(&st.minIdx, (int)i);
                atomicMax(&st.other, last);
                if (fixes) atomicMin(&st.minFix, firstFix);
                if (bads) atomicOr(&st.bad, 1);
            }
        } else {
            CellStats s = empty_stats();
            for (int d = 0; d < S.D; ++d) {
                s.lo[d] = __reduce_min_sync(grp, lo[d]);
                s.hi[d] = __reduce_max_sync(grp, hi[d]);
            }
            s.cnt = __popc(grp);
            s.minIdx = (int)i;
            s.other = last;
            s.minFix = firstFix;
            s.bad = bads != 0u;
            if (lane == leader) fold_stats(T.st + h, s, S.D, n);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kBlockCells; e += blockDim.x)
        if (B.key[e] != kEmpty && B.slot[e] >= 0) fold_stats(T.st + B.slot[e], B.st[e], S.D, n);
}

__global__ void occupied_kernel(const unsigned long long* tab, long long cap, int* occ) {
    const long long h = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (h < cap) occ[h] = tab[h] != kEmpty;
}

__global__ void cell_ids_kernel(const unsigned long long* tab, long long cap, const int* occScan, int* slotCell,
                                unsigned long long* cellKey, int* cellSlot) {
    const long long h = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= cap) return;
    if (tab[h] != kEmpty) {
        const int c = occScan[h];
        slotCell[h] = c;
        cellKey[c] = tab[h];
        cellSlot[c] = (int)h;
    } else {
        slotCell[h] = -1;
    }
}

// ---- step 2: cells -------------------------------------------------------------
struct Cells {
    int C, D;
    const unsigned long long* key;
    int* cnt;
    double* lo;  // 3 per cell
    double* hi;
    unsigned char* unsafe;  // clamped / NaN points (or eps == 0): exact point tests only
    unsigned char* dense;   // safe, and every point core
    int* minIdx;
    int* minFix;
    double* repV;  // kReps x 3 per cell
    int* repN;
    int* hasCore;  // a core point (safe cells)
    int* minCore;  // smallest core index (safe cells that are not dense)
    int* sb;       // sorted range [sb, se) (empty for a cell that was not sorted)
    int* se;
    int* need;     // to be sorted in the second pass
};

template <class Src>
__global__ void finalize_kernel(Src S, Cells K, const int* cellSlot, Table T, int compat, int zeroEps, int minPts) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= K.C) return;
    const long long h = cellSlot[c];
    const CellStats t = T.st[h];
    const int n = t.cnt;
    K.cnt[c] = n;
    for (int d = 0; d < 3; ++d) {
        K.lo[3 * c + d] = d < K.D ? (double)unfkey(t.lo[d]) : 0.0;
        K.hi[3 * c + d] = d < K.D ? (double)unfkey(t.hi[d]) : 0.0;
    }
    const bool unsafe = t.bad != 0 || zeroEps;
    const bool dense = !unsafe && (compat || n >= minPts);
    K.unsafe[c] = unsafe ? 1 : 0;
    K.dense[c] = dense ? 1 : 0;
    K.minIdx[c] = t.minIdx;
    K.minFix[c] = t.minFix;
    K.hasCore[c] = dense ? 1 : 0;
    K.minCore[c] = INT_MAX;
    K.sb[c] = 0;
    K.se[c] = 0;
    K.need[c] = 0;
    int idx[kReps], m = 0;
    idx[m++] = t.minIdx;
    if (t.other != t.minIdx) idx[m++] = t.other;
    K.repN[c] = m;
    for (int j = 0; j < m; ++j) {
        double v[3] = {0.0, 0.0, 0.0};
        S.load(idx[j], v);
        for (int d = 0; d < 3; ++d) K.repV[((long long)c * kReps + j) * 3 + d] = v[d];
    }
}

// Warp per cell: number (pass 0) or list (pass 1) of its occupied neighbour
// cells, the lanes looking up 32 of the (2R+1)^D - 1 offsets at a time (in
// the order dx, dy, dz).
__global__ void neighbours_kernel(const unsigned long long* cellKey, int C, int D, const unsigned long long* tab,
                                  unsigned long long mask, const int* slotCell, int* nbCount, const int* nbStart,
                                  int* nbList, int* nbOwner) {
    const long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (c >= C) return;
    long long base[3];
    unpack(cellKey[c], D, base);
    const int ry = D >= 2 ? kR : 0, rz = D >= 3 ? kR : 0;
    const int ny = 2 * ry + 1, nz = 2 * rz + 1, total = (2 * kR + 1) * ny * nz;
    const int w0 = nbStart ? nbStart[c] : 0;
    int k = 0;
    for (int o0 = 0; o0 < total; o0 += 32) {
        const int o = o0 + lane;
        int c2 = -1;
        if (o < total) {
            const int dz = o % nz - rz, dy = (o / nz) % ny - ry, dx = o / (nz * ny) - kR;
            if (dx != 0 || dy != 0 || dz != 0) {
                long long q[3] = {base[0] + dx, base[1] + dy, base[2] + dz};
                c2 = hash_find(tab, mask, slotCell, pack(q, D));
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, c2 >= 0);
        if (nbList && c2 >= 0) {
            const int pos = w0 + k + __popc(m & ((1u << lane) - 1u));
            nbList[pos] = c2;
            nbOwner[pos] = (int)c;
        }
        k += __popc(m);
    }
    if (!nbList && lane == 0) nbCount[c] = k;
}

// Pair states (one per neighbour entry with owner < neighbour).
enum : unsigned char {
    kFar = 0,       // boxes farther than eps apart (or the mirrored entry)
    kJoined = 1,    // settled: joined, or already in one component
    kDenseOpen = 2, // two dense cells the shortcuts did not join
    kWhole = 3,     // every point of one within eps of every point of the other (a cell not dense)
    kPoints = 4,    // point tests (a cell not dense or unsafe, boxes partly within eps)
    kDensePts = 5,  // two dense cells still apart after the shortcuts: point tests
};

__device__ __forceinline__ void pair_boxes(const Cells& K, int a, int b, double& gap2, double& span2) {
    const double* loA = K.lo + 3 * (long long)a;
    const double* hiA = K.hi + 3 * (long long)a;
    const double* loB = K.lo + 3 * (long long)b;
    const double* hiB = K.hi + 3 * (long long)b;
    gap2 = 0.0;
    span2 = 0.0;
    for (int d = 0; d < K.D; ++d) {
        double g = 0.0;
        if (hiA[d] < loB[d]) g = loB[d] - hiA[d];
        else if (hiB[d] < loA[d]) g = loA[d] - hiB[d];
        gap2 = gap2 + g * g;
        const double f = fmax(hiA[d], hiB[d]) - fmin(loA[d], loB[d]);
        span2 = span2 + f * f;
    }
}

// a representative of cell b within eps of v
__device__ __forceinline__ bool rep_within(const Cells& K, int b, const double* v, double eps) {
    for (int j = 0; j < K.repN[b]; ++j)
        if (within_eps(dist2(v, K.repV + ((long long)b * kReps + j) * 3, K.D), eps)) return true;
    return false;
}

// Thread per neighbour entry (owner < neighbour): the box tests; pairs of
// dense cells that the boxes leave open are listed for the representatives.
__global__ void pair_kernel(Cells K, const int* nbOwner, const int* nbList, double eps, unsigned char* st, int* open,
                            int* joined, int* active, unsigned char* openE, unsigned char* settledE,
                            unsigned char* deferred, int* counts) {
    const long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool take = false, join = false, act = false;
    if (w < counts[kEntries]) {
        openE[w] = settledE[w] = deferred[w] = 0;
        const int a = nbOwner[w], b = nbList[w];
        unsigned char state = kFar;
        if (b > a) {
            const double eps2 = eps * eps;
            double gap2, span2;
            pair_boxes(K, a, b, gap2, span2);
            if (gap2 > eps2 * kBoxOut) state = kFar;
            else if (K.dense[a] && K.dense[b]) {
                if (span2 < eps2 * kBoxIn) {
                    state = kJoined;  // joined by cell_components_kernel
                    join = true;
                } else {
                    state = kDenseOpen;
                    take = true;
                }
            } else {
                state = !K.unsafe[a] && !K.unsafe[b] && span2 < eps2 * kBoxIn ? kWhole : kPoints;
                act = state == kPoints;
            }
        }
        st[w] = state;
    }
    list_append(take, (int)w, open, counts + kOpen);
    list_append(join, (int)w, joined, counts + kJoinedCount);
    list_append(act, (int)w, active, counts + kActive);
}

// Warp per listed pair of dense cells: the lanes share the representative
// pairs; one within eps marks the two cells joined.
__device__ __forceinline__ void rep_pair(const Cells& K, const int* nbOwner, const int* nbList, int w, double eps,
                                         unsigned char* st, int* joined, int* nJoined) {
    const int lane = threadIdx.x & 31;
    const int a = nbOwner[w], b = nbList[w];
    const int na = K.repN[a], nb = K.repN[b];
    bool hit = false;
    for (int k = lane; k < na * nb && !hit; k += 32) {
        const double* ra = K.repV + ((long long)a * kReps + k / nb) * 3;
        const double* rb = K.repV + ((long long)b * kReps + k % nb) * 3;
        hit = within_eps(dist2(ra, rb, K.D), eps);
    }
    if (__any_sync(0xffffffffu, hit) && lane == 0) {
        st[w] = kJoined;
        joined[atomicAdd(nJoined, 1)] = w;
    }
}
__global__ void rep_pairs_kernel(Cells K, const int* nbOwner, const int* nbList, const int* open, double eps,
                                 unsigned char* st, int* joined, int* counts) {
    const int n = counts[kOpen];
    for (long long k = first_warp(); k < n; k += warp_stride())
        rep_pair(K, nbOwner, nbList, open[k], eps, st, joined, counts + kJoinedCount);
}

// The components of the dense cells over the joined pairs. Thousands of
// concurrent unions into one growing component make a global union-find
// chase pointers through L2; with up to kSharedCells cells one block runs it
// in shared memory (hooking with atomicCAS, path halving) and writes every
// cell's root, so later finds take one step. joinAll: the same over the
// global array, a thread per entry (more cells).
constexpr int kSharedCells = 40960;

__device__ __forceinline__ int sh_find(int* par, int x) {
    int cur = par[x];
    if (cur != x) {
        int prev = x, next;
        while (cur > (next = par[cur])) {
            par[prev] = next;
            prev = cur;
            cur = next;
        }
    }
    return cur;
}

__global__ void __launch_bounds__(1024) cell_components_kernel(int C, const int* nbOwner, const int* nbList,
                                                               const int* joined, const int* nJoined, int* parent) {
    extern __shared__ int par[];
    for (int v = threadIdx.x; v < C; v += blockDim.x) par[v] = v;
    __syncthreads();
    const int J = *nJoined;
    for (int k = threadIdx.x; k < J; k += blockDim.x) {
        const int e = joined[k];
        int ra = sh_find(par, nbOwner[e]), rb = sh_find(par, nbList[e]);
        while (ra != rb) {
            if (ra < rb) { const int t = ra; ra = rb; rb = t; }
            const int old = atomicCAS(par + ra, ra, rb);
            if (old == ra) break;
            ra = sh_find(par, old);
            rb = sh_find(par, rb);
        }
    }
    __syncthreads();
    for (int v = threadIdx.x; v < C; v += blockDim.x) parent[v] = sh_find(par, v);
}

__global__ void join_all_kernel(const int* nbOwner, const int* nbList, const int* joined, const int* nJoined,
                                int* parent) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < *nJoined) uf_unite(parent, nbOwner[joined[k]], nbList[joined[k]]);
}

// ---- step 3: sorting ----------------------------------------------------------
// Counting sort of the points of the cells with begin[c] >= 0 (one phase):
// one pass over the slots; only those points' features are read.
struct Sorted {
    double* s[3];
    float* r[3];  // the same relative to the lower corner of the cell's box, rounded to float (safe cells)
    int* order;
    int* cell;
    unsigned char* core;  // 0 / 1, 2 = not decided yet
    unsigned char* fix;   // reference mode
    const int* sb;
    const int* se;
    int D;
    __device__ __forceinline__ void load(int pos, double* v) const {
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (d < D) v[d] = s[d][pos];
    }
};

template <class Src>
__global__ void sort_kernel(Src S, long long n, const int* slot, const int* slotCell, const int* begin, int* cursor,
                            Sorted Q, const unsigned char* dense, int compat, const int* total) {
    if (*total == 0) return;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int h = i < n ? slot[i] : -1;
    const int c0 = h >= 0 ? slotCell[h] : -1;
    const int base = c0 >= 0 ? begin[c0] : -1;
    const int c = base >= 0 ? c0 : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, c);
    const int leader = __ffs(grp) - 1;
    int off = 0;
    if (c >= 0 && lane == leader) off = atomicAdd(&cursor[c], __popc(grp));
    off = __shfl_sync(0xffffffffu, off, leader);
    if (c < 0) return;
    const int pos = base + off + __popc(grp & ((1u << lane) - 1u));
    Q.order[pos] = (int)i;
    Q.cell[pos] = c;
    double v[3] = {0.0, 0.0, 0.0};
    S.load(i, v);
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (d < Q.D) Q.s[d][pos] = v[d];
    Q.core[pos] = compat || dense[c] ? 1 : 0;
    if (Q.fix) Q.fix[pos] = S.fix(i) ? 1 : 0;
}

__global__ void phase_begin_kernel(int C, int* scan, const int* take, const int* before, int* begin, int* sb, int* se,
                                   const int* cnt) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int offset = before ? *before : 0;
    if (take[c]) {
        begin[c] = offset + scan[c];
        sb[c] = offset + scan[c];
        se[c] = offset + scan[c] + cnt[c];
    } else {
        begin[c] = -1;
    }
    scan[c] = 0;  // from here on the sort's cursor
}

__global__ void take_sparse_kernel(Cells K, int* take) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c < K.C) take[c] = K.dense[c] ? 0 : K.cnt[c];
}

__global__ void take_needed_kernel(Cells K, int* take) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c < K.C) take[c] = K.need[c] && K.se[c] == K.sb[c] ? K.cnt[c] : 0;
}

// ---- step 3/4: point-level work on the sorted points ---------------------------------
// node of sorted point p in cell c: the cell for a safe cell, C + p otherwise
__device__ __forceinline__ int node_of(const Cells& K, int c, int p) { return K.unsafe[c] ? K.C + p : c; }

__device__ __forceinline__ bool sorted_cell(const Sorted& Q, int c) { return Q.se[c] > Q.sb[c]; }

// Long scans. A point near a dense cell that it may or may not reach has to be
// compared with the cell's points, hundreds of thousands in a map whose points
// settled on one attractor; a warp on its own would read them for
// milliseconds. Scans of safe cells of more than kLongScan points go to a
// queue instead (as long as it has room), and long_scan_kernel spreads each
// over blocks. It reads the points as float offsets from the cell's box: an
// offset is at most a few cells long and is off by less than 1e-7 of a cell,
// so a squared distance in float that is clear of eps^2 by 1e-4 decides, and
// the others are taken in FP64.
constexpr int kLongScan = 1024;
constexpr int kScanSplit = 16;  // parts of a queued scan
constexpr float kFloatOut = 1.0001f, kFloatIn = 0.9999f;

struct ScanQueue {
    int* point;
    int* cell;
    int* count;  // entries asked for; those beyond the capacity were scanned on the spot
    int cap;
    __device__ __forceinline__ bool push(int p, int c) const {  // by one lane
        if (cap == 0) return false;
        const int k = atomicAdd(count, 1);
        if (k >= cap) return false;
        point[k] = p;
        cell[k] = c;
        return true;
    }
};

// Points per block of 256 threads: the parts of the queued scans, one after
// the other. labels false: the points of the cell within eps of the point are
// counted into acc[p] until it reaches minPts. labels true: a core point
// within eps offers its component's key, the smallest wins in best[p].
__global__ void __launch_bounds__(256) long_scan_kernel(Sorted Q, Cells K, ScanQueue W, double eps, int minPts,
                                                        int labels, int* acc, unsigned long long* best, int* parent,
                                                        const int* compMin) {
    const int tasks = min(*W.count, W.cap), lane = threadIdx.x & 31;
    const float eps2 = (float)(eps * eps);
    const bool range = eps2 > 1e-30f && eps2 < 1e30f;  // else every distance is taken in FP64
    for (long long w = blockIdx.x; w < (long long)tasks * kScanSplit; w += gridDim.x) {
        const int t = (int)(w / kScanSplit), part = (int)(w % kScanSplit);
        const int p = W.point[t], c = W.cell[t];
        const int b = Q.sb[c], n = Q.se[c] - b;
        const int q0 = b + (int)((long long)n * part / kScanSplit), q1 = b + (int)((long long)n * (part + 1) / kScanSplit);
        double me[3] = {0, 0, 0};
        Q.load(p, me);
        float o[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (d < K.D) o[d] = (float)(me[d] - K.lo[3 * (long long)c + d]);
        unsigned long long key = 0;
        if (labels) {
            const int r = uf_find(parent, c);
            key = ((unsigned long long)(unsigned)compMin[r] << 32) | (unsigned)r;
        }
        const bool allCore = K.dense[c] != 0;
        int found = 0;
        constexpr int kStep = 4;  // points in flight per thread
        const int len = q1 - q0;  // (offsets from q0: a position past the part may not be an int)
        for (int q = threadIdx.x; q - (int)threadIdx.x < len; q += kStep * blockDim.x) {
            // other warps change the word: one lane reads it for its warp
            bool done = false;
            if (lane == 0) done = labels ? __ldcg(best + p) <= key : __ldcg(acc + p) >= minPts;
            if (__shfl_sync(0xffffffffu, done, 0)) break;
            float d2[kStep];
#pragma unroll
            for (int k = 0; k < kStep; ++k) {
                const int i = q + k * blockDim.x;
                d2[k] = 0.f;
                if (i < len && range) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        if (d >= K.D) continue;
                        const float df = o[d] - Q.r[d][q0 + i];
                        d2[k] = fmaf(df, df, d2[k]);
                    }
                }
            }
            int hits = 0;
#pragma unroll
            for (int k = 0; k < kStep; ++k) {
                const int i = q + k * blockDim.x;
                if (i >= len || (range && d2[k] > eps2 * kFloatOut)) continue;
                bool in = range && d2[k] < eps2 * kFloatIn;
                if (!in) {
                    double v[3];
                    Q.load(q0 + i, v);
                    in = within_eps(dist2(me, v, K.D), eps);
                }
                if (in && labels && !allCore) in = Q.core[q0 + i] == 1;
                hits += in ? 1 : 0;
            }
            found = (int)__reduce_add_sync(0xffffffffu, (unsigned)hits);
            if (found == 0) continue;
            if (lane == 0) {
                if (labels) atomicMin(best + p, key);
                else atomicAdd(acc + p, found);
            }
            if (labels) break;
        }
    }
}

// After the queued scans: the core flags of the undecided points (those marked
// 2), and their cells' links to the dense cells wholly within eps.
__device__ __forceinline__ void core_finish_point(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps,
                                   int minPts, const int* acc, int* parent, long long w) {
    const int lane = threadIdx.x & 31;
    const int p = (int)w;
    if (Q.core[p] != 2) return;
    const int c = Q.cell[p];
    const bool core = acc[p] >= minPts;
    __syncwarp();  // every lane has read the mark before lane 0 clears it
    if (lane == 0) Q.core[p] = core ? 1 : 0;
    if (!core) return;
    if (lane == 0 && !K.unsafe[c]) {
        atomicOr(&K.hasCore[c], 1);
        atomicMin(&K.minCore[c], Q.order[p]);
    }
    double me[3] = {0, 0, 0};
    Q.load(p, me);
    const double eps2 = eps * eps;
    for (int e = nbStart[c] + lane; e < nbStart[c + 1]; e += 32) {
        const int b = nbList[e];
        if (K.unsafe[b] || !K.dense[b]) continue;
        double near2, far2;
        box_dist2(me, K.lo + 3 * (long long)b, K.hi + 3 * (long long)b, K.D, near2, far2);
        if (near2 <= eps2 * kBoxOut && far2 < eps2 * kBoxIn) uf_unite(parent, node_of(K, c, p), b);
    }
}

__global__ void core_finish_kernel(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps,
                                   int minPts, const int* acc, int* parent, const int* counts) {
    const int n = counts[kSparse];
    for (long long w = first_warp(); w < n; w += warp_stride())
        core_finish_point(Q, K, nbStart, nbList, eps, minPts, acc, parent, w);
}

// Warp per sorted point of a cell that is not dense (textbook mode), in
// [0, M1): the lanes classify the neighbour cells (at most 124, four per
// lane) by their boxes -- beyond eps: nothing; wholly within eps: counted
// whole; partly: scanned if sorted, otherwise (a dense cell) its
// representatives within eps counted, a lower bound -- then the sorted cells
// are scanned 32 points at a time until minPts. A point that stays below
// minPts with a lower-bound cell is left undecided (core = 2) and those cells
// are marked for the second sort. redo: only the undecided points, counted
// exactly into acc, long scans through the queue; core_finish_kernel decides.
constexpr int kNbPerLane = 4;  // (2R+1)^3 - 1 = 124 neighbour cells at most

__device__ __forceinline__ void core_point(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps, int minPts,
                            int redo, ScanQueue W, int* acc, long long w) {
    const int lane = threadIdx.x & 31;
    const int p = (int)w;
    if (redo && Q.core[p] != 2) return;
    const int c = Q.cell[p];
    double me[3] = {0, 0, 0};
    Q.load(p, me);
    const double eps2 = eps * eps;
    const int e0 = nbStart[c], e1 = nbStart[c + 1];
    int cls[kNbPerLane];  // 0 nothing, 1 whole, 2 scan, 3 representatives (a lower bound)
    int local = 0;
    bool lower = false;
#pragma unroll
    for (int j = 0; j < kNbPerLane; ++j) {
        const int e = e0 + lane + 32 * j;
        cls[j] = 0;
        if (e >= e1) continue;
        const int b = nbList[e];
        if (K.unsafe[b]) {
            cls[j] = 2;
            continue;
        }
        double near2, far2;
        box_dist2(me, K.lo + 3 * (long long)b, K.hi + 3 * (long long)b, K.D, near2, far2);
        if (near2 > eps2 * kBoxOut) continue;
        if (far2 < eps2 * kBoxIn) {
            cls[j] = 1;
            local += K.cnt[b];
            continue;
        }
        if (sorted_cell(Q, b)) {
            cls[j] = 2;
            continue;
        }
        cls[j] = 3;
        lower = true;
        for (int r = 0; r < K.repN[b]; ++r)
            if (within_eps(dist2(me, K.repV + ((long long)b * kReps + r) * 3, K.D), eps)) ++local;
    }
    int cnt = (K.unsafe[c] ? 0 : K.cnt[c]) + (int)__reduce_add_sync(0xffffffffu, (unsigned)local);
    const bool inexact = __any_sync(0xffffffffu, lower);
    auto scan_cell = [&](int cell) {
        const int end = Q.se[cell];
        for (int q0 = Q.sb[cell]; q0 < end && cnt < minPts; q0 += 32) {
            const int q = q0 + lane;
            bool hit = false;
            if (q < end) {
                double v[3];
                Q.load(q, v);
                hit = within_eps(dist2(me, v, K.D), eps);
            }
            cnt += __popc(__ballot_sync(0xffffffffu, hit));
        }
    };
    if (K.unsafe[c] && cnt < minPts) scan_cell(c);
    unsigned queued[kNbPerLane];  // long scans left to the queue (redo)
#pragma unroll
    for (int j = 0; j < kNbPerLane; ++j) {
        unsigned m = __ballot_sync(0xffffffffu, cls[j] == 2);
        queued[j] = 0;
        while (m && cnt < minPts) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const int b = nbList[e0 + src + 32 * j];
            if (redo && !K.unsafe[b] && Q.se[b] - Q.sb[b] > kLongScan) queued[j] |= 1u << src;
            else scan_cell(b);
        }
    }
    if (redo) {  // core_finish_kernel decides, after the queued scans
        bool full = false;
        if (lane == 0) acc[p] = cnt;
#pragma unroll
        for (int j = 0; j < kNbPerLane; ++j)
            while (queued[j] && cnt < minPts) {
                const int src = __ffs(queued[j]) - 1;
                queued[j] &= queued[j] - 1;
                const int b = nbList[e0 + src + 32 * j];
                if (!full) full = __shfl_sync(0xffffffffu, lane == 0 && !W.push(p, b), 0);
                if (full) {
                    const int before = cnt;
                    scan_cell(b);
                    if (lane == 0) atomicAdd(acc + p, cnt - before);
                }
            }
        return;
    }
    const int core = cnt >= minPts ? 1 : (inexact ? 2 : 0);
    if (lane == 0) {
        Q.core[p] = (unsigned char)core;
        if (core == 1 && !K.unsafe[c]) {
            atomicOr(&K.hasCore[c], 1);
            atomicMin(&K.minCore[c], Q.order[p]);
        }
    }
#pragma unroll
    for (int j = 0; j < kNbPerLane; ++j)
        if (cls[j] == 3 && core == 2) K.need[nbList[e0 + lane + 32 * j]] = 1;  // to be sorted
}

__global__ void core_kernel(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps, int minPts,
                            int redo, ScanQueue W, int* acc, const int* counts) {
    const int n = counts[kSparse];
    for (long long w = first_warp(); w < n; w += warp_stride())
        core_point(Q, K, nbStart, nbList, eps, minPts, redo, W, acc, w);
}

// Warp per sorted point of a cell that is not dense, in [0, M1), after the
// core flags, lanes over the neighbour cells: a core point of a safe cell
// joins its cell to every dense neighbour that is whole within eps of it or
// holds a representative within eps; an entry (cell -> dense neighbour) that
// none of the cell's core points settled that way is marked open. A point
// that is not core marks the dense neighbours its border label would have to
// scan (partly within eps, no representative within eps), and a point of an
// unsafe cell every dense neighbour within reach: those are sorted in the
// second pass.
__device__ __forceinline__ void dense_links_point(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps,
                                   int* parent, unsigned char* openE, unsigned char* settledE, long long w) {
    const int lane = threadIdx.x & 31;
    const int p = (int)w;
    const int c = Q.cell[p];
    const int core = Q.core[p];
    if (core == 2) return;  // its neighbours are sorted in the second pass
    double me[3] = {0, 0, 0};
    Q.load(p, me);
    const double eps2 = eps * eps;
    for (int e = nbStart[c] + lane; e < nbStart[c + 1]; e += 32) {
        const int b = nbList[e];
        if (!K.dense[b]) continue;
        double near2, far2;
        box_dist2(me, K.lo + 3 * (long long)b, K.hi + 3 * (long long)b, K.D, near2, far2);
        if (near2 > eps2 * kBoxOut) continue;
        if (K.unsafe[c]) {
            K.need[b] = 1;
            continue;
        }
        const bool reach = far2 < eps2 * kBoxIn || rep_within(K, b, me, eps);
        if (core == 1) {
            if (reach) {
                uf_unite(parent, c, b);
                settledE[e] = 1;
            } else {
                openE[e] = 1;
            }
        } else if (!reach) {
            K.need[b] = 1;
        }
    }
}

__global__ void dense_links_kernel(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps,
                                   int* parent, unsigned char* openE, unsigned char* settledE, const int* counts) {
    const int n = counts[kSparse];
    for (long long w = first_warp(); w < n; w += warp_stride())
        dense_links_point(Q, K, nbStart, nbList, eps, parent, openE, settledE, w);
}

// Entry pass after the shortcuts' unions: two dense cells still apart, and
// open entries of a cell whose core points did not reach a dense neighbour,
// get point tests (both cells sorted) when they are in two components; pairs
// with an unsafe cell are tested point by point.
__global__ void open_pairs_kernel(Cells K, const int* nbOwner, const int* nbList, int* parent, unsigned char* st,
                                  const unsigned char* openE, const unsigned char* settledE, int* active, int* counts) {
    const long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= counts[kEntries]) return;
    const int a = nbOwner[w], b = nbList[w];
    if (st[w] == kDenseOpen) {
        if (uf_find(parent, a) != uf_find(parent, b)) {
            st[w] = kDensePts;
            active[atomicAdd(counts + kActive, 1)] = (int)w;
            K.need[a] = 1;
            K.need[b] = 1;
        } else {
            st[w] = kJoined;
        }
    }
    if (openE[w] && !settledE[w] && uf_find(parent, a) != uf_find(parent, b)) K.need[b] = 1;
    if (st[w] == kPoints && (K.unsafe[a] || K.unsafe[b])) {
        K.need[a] = 1;
        K.need[b] = 1;
    }
}

// ---- step 5: unions ------------------------------------------------------------

__global__ void whole_pairs_kernel(Cells K, const int* nbOwner, const int* nbList, const unsigned char* st, int* parent,
                                   const int* counts) {
    const long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= counts[kEntries] || st[w] != kWhole) return;
    const int a = nbOwner[w], b = nbList[w];
    if (K.hasCore[a] && K.hasCore[b]) uf_unite(parent, a, b);
}

// warp per unsafe cell: exact pair tests between its core points
__global__ void unsafe_cell_kernel(Sorted Q, Cells K, double eps, int* parent) {
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= K.C || !K.unsafe[w]) return;
    const int b = Q.sb[w], e = Q.se[w];
    for (int p = b; p < e; ++p) {
        if (Q.core[p] != 1) continue;
        double a[3];
        Q.load(p, a);
        for (int q = p + 1 + lane; q < e; q += 32) {
            if (Q.core[q] != 1) continue;
            double v[3];
            Q.load(q, v);
            if (within_eps(dist2(a, v, K.D), eps)) uf_unite(parent, K.C + p, K.C + q);
        }
    }
}

// warp per listed entry (state kPoints / kDensePts) whose two cells are sorted:
// unite the two cells' core points if any core pair is within eps. The
// smaller cell's points are walked one by one, the larger cell's 32 at a
// time.
//
// Three passes of growing budget. Pass 0 probes every pair with a small
// amount of work (kPassOuter points of the smaller cell against kPassChunks
// x 32 points of the larger one) and marks the pairs it could not settle;
// each later pass takes the marked pairs only, first skips those whose two
// cells earlier unions already put into one component, and the last pass
// scans exhaustively. The components found do not depend on the order of
// the unions.
constexpr int kCrossPasses = 3;
__constant__ int kPassOuter[kCrossPasses] = {2, 32, 0x7fffffff};
__constant__ int kPassChunks[kCrossPasses] = {2, 8, 0x7fffffff};

constexpr long long kLongPair = 1 << 16;  // point pairs of two cells that one warp takes on in the last pass

__device__ __forceinline__ void cross_cells(Sorted Q, Cells K, const int* nbOwner, const int* nbList, double eps,
                                            int* parent, int pass, unsigned char* deferred, int* longPairs, int* nLong,
                                            long long w) {
    const int lane = threadIdx.x & 31;
    int ca = nbOwner[w], cb = nbList[w];
    if (!sorted_cell(Q, ca) || !sorted_cell(Q, cb)) return;
    const bool last = pass == kCrossPasses - 1;
    if (pass > 0) {
        const bool todo = deferred[w] != 0;
        __syncwarp();  // every lane has read the mark before lane 0 clears it
        if (!todo) return;
        if (lane == 0) deferred[w] = 0;
    }
    const bool safe = !K.unsafe[ca] && !K.unsafe[cb];
    if (safe && (!K.hasCore[ca] || !K.hasCore[cb])) return;
    if (!safe && !last) {  // unsafe cells unite every core pair within eps: last pass only
        if (lane == 0) deferred[w] = 1;
        return;
    }
    if (safe) {  // other warps unite cells meanwhile: one lane looks for its warp
        bool joined = false;
        if (lane == 0) joined = uf_find(parent, ca) == uf_find(parent, cb);
        if (__shfl_sync(0xffffffffu, joined, 0)) return;
    }
    const double eps2 = eps * eps;
    double gap2, span2;
    pair_boxes(K, ca, cb, gap2, span2);
    if (gap2 > eps2 * kBoxOut) return;
    if (Q.se[ca] - Q.sb[ca] > Q.se[cb] - Q.sb[cb]) {
        const int t = ca;
        ca = cb;
        cb = t;
    }
    if (last && safe && (long long)(Q.se[ca] - Q.sb[ca]) * (Q.se[cb] - Q.sb[cb]) > kLongPair) {
        if (lane == 0) longPairs[atomicAdd(nLong, 1)] = (int)w;  // long_pairs_kernel
        return;
    }
    const double* lo = K.lo + 3 * (long long)cb;
    const double* hi = K.hi + 3 * (long long)cb;
    int outerLeft = kPassOuter[pass];
    const int chunkBudget = kPassChunks[pass];
    bool cut = false, stop = false;
    const int endA = Q.se[ca], endB = Q.se[cb];
    for (int p0 = Q.sb[ca]; p0 < endA && !stop; p0 += 32) {
        const int p = p0 + lane;
        double a[3] = {0, 0, 0};
        bool inReach = false, allIn = false;
        if (p < endA && Q.core[p] == 1) {
            Q.load(p, a);
            double near2, far2;
            box_dist2(a, lo, hi, K.D, near2, far2);
            inReach = near2 <= eps2 * kBoxOut;
            allIn = safe && far2 < eps2 * kBoxIn;
        }
        const unsigned mAll = __ballot_sync(0xffffffffu, inReach && allIn);
        if (mAll) {  // every core point of cb is within eps of this one
            if (lane == __ffs(mAll) - 1) uf_unite(parent, ca, cb);
            return;
        }
        unsigned todo = __ballot_sync(0xffffffffu, inReach);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            if (outerLeft-- == 0) {
                cut = stop = true;
                break;
            }
            const int pp = p0 + src;
            double aa[3];
            for (int d = 0; d < 3; ++d) aa[d] = __shfl_sync(0xffffffffu, a[d], src);
            int chunks = 0;
            for (int q0 = Q.sb[cb]; q0 < endB; q0 += 32) {
                if (chunks++ == chunkBudget) {
                    cut = true;
                    break;
                }
                const int q = q0 + lane;
                bool hit = false;
                if (q < endB && Q.core[q] == 1) {
                    double v[3];
                    Q.load(q, v);
                    hit = within_eps(dist2(aa, v, K.D), eps);
                }
                const unsigned bal = __ballot_sync(0xffffffffu, hit);
                if (bal) {
                    if (safe) {
                        if (lane == __ffs(bal) - 1) uf_unite(parent, ca, cb);
                        return;
                    }
                    if (hit) uf_unite(parent, node_of(K, ca, pp), node_of(K, cb, q));
                }
            }
        }
    }
    if (cut && lane == 0) deferred[w] = 1;
}

__global__ void cross_cell_kernel(Sorted Q, Cells K, const int* nbOwner, const int* nbList, double eps, int* parent,
                                  int pass, unsigned char* deferred, int* longPairs, int* nLong, const int* active,
                                  const int* counts) {
    const int n = counts[kActive];
    for (long long k = first_warp(); k < n; k += warp_stride())
        cross_cells(Q, K, nbOwner, nbList, eps, parent, pass, deferred, longPairs, nLong, active[k]);
}

// The listed pairs of safe cells that the passes left apart and whose points
// make more than kLongPair pairs: the larger cell's points, a block of them
// at a time, against all of the smaller cell's, as long as the two are in two
// components. One warp for a whole pair took 9.5 ms where a few points face a
// cell of 250,000 just out of reach. Distances as in long_scan_kernel.
__global__ void __launch_bounds__(256) long_pairs_kernel(Sorted Q, Cells K, const int* nbOwner, const int* nbList,
                                                         const int* longPairs, const int* nLong, double eps,
                                                         int* parent) {
    __shared__ float so[3][256];
    __shared__ int apart;
    const int n = *nLong;
    const float eps2 = (float)(eps * eps);
    const bool range = eps2 > 1e-30f && eps2 < 1e30f;
    // all blocks on one pair, or at least 16 on each of many
    const int team = n > 0 ? max(16, (int)gridDim.x / n) : 1, teams = max(1, (int)gridDim.x / team);
    if ((int)blockIdx.x >= team * teams) return;
    for (int t = blockIdx.x / team; t < n; t += teams) {
        int ca = nbOwner[longPairs[t]], cb = nbList[longPairs[t]];
        if (Q.se[ca] - Q.sb[ca] > Q.se[cb] - Q.sb[cb]) {
            const int x = ca;
            ca = cb;
            cb = x;
        }
        const double* lo = K.lo + 3 * (long long)cb;
        const bool coreA = K.dense[ca] != 0, coreB = K.dense[cb] != 0;
        const int endA = Q.se[ca], endB = Q.se[cb];
        // (64 bits: a block past the last one may not have an int for its start)
        for (long long q0 = Q.sb[cb] + (long long)(blockIdx.x % team) * 256; q0 < endB; q0 += team * 256) {
            __syncthreads();
            if (threadIdx.x == 0) apart = uf_find(parent, ca) != uf_find(parent, cb);
            __syncthreads();
            if (!apart) break;
            const long long q = q0 + threadIdx.x;
            const bool mine = q < endB && (coreB || Q.core[q] == 1);
            float r[3] = {0.f, 0.f, 0.f};
            if (mine) {
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    if (d < K.D) r[d] = Q.r[d][q];
            }
            bool hit = false;
            for (long long p0 = Q.sb[ca]; p0 < endA; p0 += 256) {
                const long long p = p0 + threadIdx.x;
                __syncthreads();
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    if (d >= K.D) continue;
                    so[d][threadIdx.x] = p < endA && (coreA || Q.core[p] == 1) ? (float)(Q.s[d][p] - lo[d])
                                                                              : __int_as_float(0x7f800000);
                }
                __syncthreads();
                const int m = (int)min(256LL, endA - p0);
                for (int k = 0; k < m && mine && !hit; ++k) {
                    float sum = 0.f;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        if (d >= K.D) continue;
                        const float df = r[d] - so[d][k];
                        sum = fmaf(df, df, sum);
                    }
                    if (sum > eps2 * kFloatOut && (range || sum == __int_as_float(0x7f800000))) continue;
                    if (range && sum < eps2 * kFloatIn) {
                        hit = true;
                        continue;
                    }
                    double a[3] = {0, 0, 0}, b[3] = {0, 0, 0};
                    Q.load((int)p0 + k, a);
                    Q.load((int)q, b);
                    hit = (coreA || Q.core[p0 + k] == 1) && within_eps(dist2(a, b, K.D), eps);
                }
                if (__syncthreads_or(hit)) break;
            }
            if (hit) uf_unite(parent, ca, cb);
        }
    }
}

// ---- step 6: components and labels ------------------------------------------------
__global__ void iota_kernel(int* p, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = (int)i;
}

// The nodes of the final union-find: the cells' components so far, then the
// sorted points (and their offsets from their cells' boxes).
__global__ void nodes_kernel(Sorted Q, Cells K, const int* parentC, int* parent, int* compMin, int* compFix,
                             const int* counts) {
    const long long n = (long long)K.C + sorted_points(counts);
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        parent[v] = v < K.C ? parentC[v] : (int)v;
        compMin[v] = INT_MAX;
        compFix[v] = INT_MAX;
        if (v < K.C) continue;
        const long long p = v - K.C, c = Q.cell[p];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (d < Q.D) Q.r[d][p] = (float)(Q.s[d][p] - K.lo[3 * c + d]);
    }
}

// node's smallest core (and fixed-point) index, folded into its component's root
__device__ __forceinline__ bool node_keys(const Sorted& Q, const Cells& K, int v, int& key, int& fixKey) {
    if (v < K.C) {
        if (K.unsafe[v] || !K.hasCore[v]) return false;
        key = K.dense[v] ? K.minIdx[v] : K.minCore[v];
        fixKey = K.minFix[v];
        return true;
    }
    const int p = v - K.C;
    if (!K.unsafe[Q.cell[p]] || Q.core[p] != 1) return false;
    key = Q.order[p];
    fixKey = Q.fix && Q.fix[p] ? Q.order[p] : INT_MAX;
    return true;
}

__global__ void comp_kernel(Sorted Q, Cells K, int* parent, int* compMin, int* compFix, const int* counts) {
    const long long n = (long long)K.C + sorted_points(counts);
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        int key, fixKey;
        if (!node_keys(Q, K, (int)v, key, fixKey)) continue;
        const int r = uf_find(parent, (int)v);
        atomicMin(&compMin[r], key);
        if (fixKey != INT_MAX) atomicMin(&compFix[r], fixKey);
    }
}

// Numbering: textbook, the components by their smallest core index; reference
// mode, those with a fixed point by their smallest fixed-point index (-1, -2,
// ...), the others by their smallest index. Each root marks its index in a bit
// array over the points (fixed-point components in a second one), whose prefix
// sums rank it.
__global__ void root_marks_kernel(Sorted Q, Cells K, int* parent, const int* compMin, const int* compFix, int compat,
                                  unsigned* bits, unsigned* fixBits, const int* counts) {
    const long long n = (long long)K.C + sorted_points(counts);
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        int key, fixKey;
        if (!node_keys(Q, K, (int)v, key, fixKey) || uf_find(parent, (int)v) != (int)v) continue;
        const bool fix = compat && compFix[v] != INT_MAX;
        const int at = fix ? compFix[v] : compMin[v];
        atomicOr((fix ? fixBits : bits) + (at >> 5), 1u << (at & 31));
    }
}

__global__ void bit_counts_kernel(const unsigned* bits, int* cnt, long long words) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < words) cnt[i] = __popc(bits[i]);
}

__global__ void root_labels_kernel(Sorted Q, Cells K, int* parent, const int* compMin, const int* compFix, int compat,
                                   const unsigned* bits, const unsigned* fixBits, const int* rank, const int* fixRank,
                                   int* compLabel, const int* counts) {
    const long long n = (long long)K.C + sorted_points(counts);
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        int key, fixKey;
        if (!node_keys(Q, K, (int)v, key, fixKey) || uf_find(parent, (int)v) != (int)v) continue;
        const bool fix = compat && compFix[v] != INT_MAX;
        const int at = fix ? compFix[v] : compMin[v];
        const int r = (fix ? fixRank : rank)[at >> 5] + __popc((fix ? fixBits : bits)[at >> 5] & ((1u << (at & 31)) - 1u));
        compLabel[v] = fix ? -(r + 1) : (compat ? r + 1 : r);
    }
}

__global__ void cell_labels_kernel(Cells K, int* parent, const int* compLabel, int* cellLabel) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= K.C) return;
    cellLabel[c] = !K.unsafe[c] && K.hasCore[c] ? compLabel[uf_find(parent, (int)c)] : -1;
}

// one pass over the slots: excluded points, and every point of a dense cell
__global__ void labels_kernel(const int* slot, const int* slotCell, long long n, const unsigned char* dense,
                              const int* cellLabel, int compat, int* labels) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int h = slot[i];
    if (h < 0) {
        labels[i] = compat ? 0 : -2;
        return;
    }
    const int c = slotCell[h];
    if (dense[c]) labels[i] = cellLabel[c];
}

// Warp per sorted point of a cell that is not dense, in [0, M1): a core
// point takes its component's label; a border point the component with the
// smallest core index among the core points within eps (lanes settle the
// neighbour cells by box or representatives, the rest are scanned by the
// warp or, the long ones, through the queue, a safe cell only while it could
// still lower the answer); the rest are noise (-1). border_labels_kernel
// writes those that are not core.
__device__ __forceinline__ void sorted_label(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps,
                                     int* parent, const int* compMin, const int* compLabel, int* labels, ScanQueue W,
                                     unsigned long long* bests, long long w) {
    const int lane = threadIdx.x & 31;
    const int p = (int)w;
    const int c = Q.cell[p];
    if (Q.core[p] == 1) {
        if (lane == 0) labels[Q.order[p]] = compLabel[uf_find(parent, node_of(K, c, p))];
        return;
    }
    double me[3] = {0, 0, 0};
    Q.load(p, me);
    const double eps2 = eps * eps;
    const int e0 = nbStart[c], e1 = nbStart[c + 1];
    // candidates as (smallest core index of the component, root): the smallest wins
    auto key_of = [&](int r) { return ((unsigned long long)(unsigned)compMin[r] << 32) | (unsigned)r; };
    unsigned long long best = ~0ull;
    if (lane == 0 && !K.unsafe[c] && K.hasCore[c]) best = key_of(uf_find(parent, c));  // own cell: within eps
    bool scanIt[kNbPerLane];
#pragma unroll
    for (int j = 0; j < kNbPerLane; ++j) {
        const int e = e0 + lane + 32 * j;
        scanIt[j] = false;
        if (e >= e1) continue;
        const int b = nbList[e];
        if (K.unsafe[b]) {
            scanIt[j] = true;
            continue;
        }
        if (!K.hasCore[b]) continue;
        double near2, far2;
        box_dist2(me, K.lo + 3 * (long long)b, K.hi + 3 * (long long)b, K.D, near2, far2);
        if (near2 > eps2 * kBoxOut) continue;
        if (far2 < eps2 * kBoxIn || (K.dense[b] && rep_within(K, b, me, eps))) {
            const unsigned long long k = key_of(uf_find(parent, b));
            best = k < best ? k : best;
            continue;
        }
        scanIt[j] = true;  // sorted: a dense cell here was marked for the second pass
    }
    best = group_min64(0xffffffffu, best);
    auto scan = [&](int cell) {
        const int end = Q.se[cell];
        if (!K.unsafe[cell]) {  // all its core points share one root
            const unsigned long long k = key_of(uf_find(parent, cell));
            if (k >= best) return;
            for (int q0 = Q.sb[cell]; q0 < end; q0 += 32) {
                const int q = q0 + lane;
                bool hit = false;
                if (q < end && Q.core[q] == 1) {
                    double v[3];
                    Q.load(q, v);
                    hit = within_eps(dist2(me, v, K.D), eps);
                }
                if (__any_sync(0xffffffffu, hit)) {
                    best = k;
                    return;
                }
            }
            return;
        }
        for (int q0 = Q.sb[cell]; q0 < end; q0 += 32) {
            const int q = q0 + lane;
            unsigned long long k = ~0ull;
            if (q < end && Q.core[q] == 1) {
                double v[3];
                Q.load(q, v);
                if (within_eps(dist2(me, v, K.D), eps)) k = key_of(uf_find(parent, node_of(K, cell, q)));
            }
            k = group_min64(0xffffffffu, k);
            best = k < best ? k : best;
        }
    };
    if (K.unsafe[c]) scan(c);
    bool full = false;
    unsigned queued[kNbPerLane];  // long scans left to the queue
#pragma unroll
    for (int j = 0; j < kNbPerLane; ++j) {
        unsigned m = __ballot_sync(0xffffffffu, scanIt[j]);
        queued[j] = 0;
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const int b = nbList[e0 + src + 32 * j];
            if (!K.unsafe[b] && Q.se[b] - Q.sb[b] > kLongScan) queued[j] |= 1u << src;
            else scan(b);
        }
    }
    if (lane == 0) bests[p] = best;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kNbPerLane; ++j)
        while (queued[j]) {
            const int src = __ffs(queued[j]) - 1;
            queued[j] &= queued[j] - 1;
            const int b = nbList[e0 + src + 32 * j];
            if (key_of(uf_find(parent, b)) >= best) continue;  // could not lower the answer
            if (!full) full = __shfl_sync(0xffffffffu, lane == 0 && !W.push(p, b), 0);
            if (full) {
                scan(b);
                if (lane == 0) atomicMin(bests + p, best);
            }
        }
}

__global__ void sorted_labels_kernel(Sorted Q, Cells K, const int* nbStart, const int* nbList, double eps,
                                     int* parent, const int* compMin, const int* compLabel, int* labels, ScanQueue W,
                                     unsigned long long* bests, const int* counts) {
    const int n = counts[kSparse];
    for (long long w = first_warp(); w < n; w += warp_stride())
        sorted_label(Q, K, nbStart, nbList, eps, parent, compMin, compLabel, labels, W, bests, w);
}

// After the queued scans: the labels of the points that are not core.
__global__ void border_labels_kernel(Sorted Q, const unsigned long long* bests, const int* compLabel, int* labels,
                                     const int* counts) {
    const int n = counts[kSparse];
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        if (Q.core[p] == 1) continue;
        const unsigned long long best = bests[p];
        labels[Q.order[p]] = best == ~0ull ? -1 : compLabel[(int)(best & 0xffffffffull)];
    }
}

#define CK(x)                                                   \
    do {                                                        \
        cudaError_t e_ = (x);                                   \
        if (e_ != cudaSuccess) return cuda_error(e_, #x);       \
    } while (0)
#define CKL() CK(cudaGetLastError())
#define NEED(p) \
    if (!(p)) return CHAOS_E_NOMEM

// Scratch arrays of one call, several to an allocation.
struct Arena {
    Call& c;
    char* at = nullptr;
    size_t left = 0;
    template <class T> T* take(size_t count) {
        const size_t bytes = (count * sizeof(T) + 255) / 256 * 256;
        if (bytes > left) {
            constexpr size_t kChunk = 4 << 20;
            char* p = (char*)c.alloc(std::max(bytes, kChunk));
            if (!p) return nullptr;
            if (bytes >= kChunk) return (T*)p;
            at = p;
            left = kChunk;
        }
        T* r = (T*)at;
        at += bytes;
        left -= bytes;
        return r;
    }
};

// The pipeline. compat: the reference's eps-components (every included point
// core, numbering by fixed points); otherwise textbook DBSCAN with minPts.
// bound > 0: a bound on the occupied cells known from the source. Without one,
// a small set's table is sized by its points (measuring their extent takes a
// pass and a wait, more than the larger table costs), a large one's by the
// extent of its cells. Every wait for a count costs the host's round trip and
// an idle GPU. Of seven, small sets keep one (the cells), sets above kSmallSet
// one more (the extent; a basin map brings its bound), more than 8,456 cells in
// 3-D (43,690 in 2-D) one more (their neighbour entries) and sets above
// kRoomySet one more (the sorted points): with that, and the scratch in few
// allocations, 10,000 points take 256 instead of 445 us, 1,000,000 505 instead of
// 690. Fout (basin maps) receives the normalised features.
constexpr long long kSmallSet = 65536;
constexpr long long kRoomySet = 1 << 22;  // beyond it, 36 B of scratch a point are worth a wait

template <class Src>
int cell_cluster(Call& c, const Src& S, long long n, double eps, int minPts, bool compat, double bound, double* Fout,
                 int* labels) {
    cudaStream_t st = c.stream;
    const int D = S.D;
    const bool zeroEps = !(eps > 0);
    const double side = zeroEps ? 1.0 : eps / sqrt((double)D) * (1.0 - 1e-9);
    const double invSide = 1.0 / side;
    int sms = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
    sms = std::max(sms, 1);
    const unsigned loop = (unsigned)(kLoopBlocksPerSm * sms);
    Arena A{c};
    int* counts = A.take<int>(kCounts);
    NEED(counts);
    CK(cudaMemsetAsync(counts, 0, kCounts * sizeof(int), st));
    if (!(bound > 0) && n > kSmallSet) {
        long long* ext = A.take<long long>(8);
        NEED(ext);
        const long long init[8] = {LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN, 0, 0};
        CK(cudaMemcpyAsync(ext, init, sizeof init, cudaMemcpyHostToDevice, st));
        extent_kernel<Src><<<blocks(n), kTPB, 0, st>>>(S, n, invSide, ext);
        note_launch();
        long long hx[8];
        CK(cudaMemcpyAsync(hx, ext, sizeof hx, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        bound = (double)hx[6];
        if (hx[3] != LLONG_MIN) {  // some ordinary point
            double prod = 1.0;
            for (int d = 0; d < D; ++d) prod *= (double)(hx[3 + d] + hx[d] + 1);
            bound += prod;
        }
    } else if (!(bound > 0)) {
        bound = (double)n;
    }
    bound = std::min(bound, (double)n);
    unsigned long long cap = 1024;
    while ((double)cap < 2.0 * bound + 2.0) cap <<= 1;
    Table T;
    T.mask = cap - 1;
    T.key = A.take<unsigned long long>(cap);
    T.st = A.take<CellStats>(cap);
    int* slot = A.take<int>(n);
    int* occ = A.take<int>(cap);
    int* slotCell = A.take<int>(cap);
    NEED(!c.failed);
    table_init_kernel<<<blocks(cap), kTPB, 0, st>>>(T, (long long)cap);
    note_launch();
    {
        const long long most = (long long)sms * kCellBlocksPerSm;
        const long long rows = (n + kCellBlock - 1) / kCellBlock, per = (rows + most - 1) / most;
        CK(cudaFuncSetAttribute(cells_kernel<Src>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BlockCells)));
        cells_kernel<Src><<<(unsigned)((rows + per - 1) / per), kCellBlock, sizeof(BlockCells), st>>>(
            S, n, per * kCellBlock, invSide, T, slot, Fout, counts + kErr);
        note_launch();
    }
    occupied_kernel<<<blocks(cap), kTPB, 0, st>>>(T.key, cap, occ);
    note_launch();
    CKL();
    int rc = device_scan(c, occ, occ, (long long)cap, counts + kCells);
    if (rc) return rc;
    int hc[2] = {0, 0};
    static_assert(kErr == kCells + 1, "read together");
    CK(cudaMemcpyAsync(hc, counts + kCells, sizeof hc, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (hc[1]) return set_error(CHAOS_E_CUDA, "clustering: cell table full");
    const int C = hc[0];
    Cells K;
    K.C = C;
    K.D = D;
    const size_t C1 = (size_t)C + 1;
    unsigned long long* cellKey = A.take<unsigned long long>(C1);
    int* cellSlot = A.take<int>(C1);
    K.key = cellKey;
    K.cnt = A.take<int>(C1);
    K.lo = A.take<double>(3 * C1);
    K.hi = A.take<double>(3 * C1);
    K.unsafe = A.take<unsigned char>(C1);
    K.dense = A.take<unsigned char>(C1);
    K.minIdx = A.take<int>(C1);
    K.minFix = A.take<int>(C1);
    K.repV = A.take<double>(C1 * kReps * 3);
    K.repN = A.take<int>(C1);
    K.hasCore = A.take<int>(C1);
    K.minCore = A.take<int>(C1);
    K.sb = A.take<int>(C1);
    K.se = A.take<int>(C1);
    K.need = A.take<int>(C1);
    int* nbStart = A.take<int>(C1);
    int* take = A.take<int>(C1);
    int* begin = A.take<int>(C1);
    int* cursor = A.take<int>(C1);
    int* parentC = A.take<int>(C1);
    int* cellLabel = A.take<int>(C1);
    NEED(!c.failed);
    if (C == 0) {  // no point takes part
        labels_kernel<<<blocks(n), kTPB, 0, st>>>(slot, slotCell, n, K.dense, cellLabel, compat ? 1 : 0, labels);
        note_launch();
        CKL();
        return CHAOS_OK;
    }
    cell_ids_kernel<<<blocks(cap), kTPB, 0, st>>>(T.key, cap, occ, slotCell, cellKey, cellSlot);
    note_launch();
    finalize_kernel<Src><<<blocks(C), kTPB, 0, st>>>(S, K, cellSlot, T, compat ? 1 : 0, zeroEps ? 1 : 0, minPts);
    note_launch();
    neighbours_kernel<<<blocks((long long)C * 32), kTPB, 0, st>>>(cellKey, C, D, T.key, T.mask, slotCell, nbStart,
                                                                  nullptr, nullptr, nullptr);
    note_launch();
    iota_kernel<<<blocks(C), kTPB, 0, st>>>(parentC, C);
    note_launch();
    CKL();
    CK(cudaMemsetAsync(nbStart + C, 0, sizeof(int), st));
    if ((rc = device_scan(c, nbStart, nbStart, (long long)C + 1, counts + kEntries))) return rc;
    // room for the neighbour entries: by their bound while that is small,
    // otherwise by their number, which takes a wait
    long long E = (long long)C * (D == 1 ? 2 * kR : (D == 2 ? 24 : 124));
    if (E > (1 << 20)) {
        int hE = 0;
        CK(cudaMemcpyAsync(&hE, counts + kEntries, sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        E = hE;
    }
    const size_t E1 = (size_t)E + 1;
    int* nbList = A.take<int>(E1);
    int* nbOwner = A.take<int>(E1);
    unsigned char* pst = A.take<unsigned char>(E1);
    unsigned char* openE = A.take<unsigned char>(E1);
    unsigned char* settledE = A.take<unsigned char>(E1);
    unsigned char* deferred = A.take<unsigned char>(E1);
    int* openList = A.take<int>(E1);
    int* joinList = A.take<int>(E1);
    int* active = A.take<int>(E1);
    NEED(!c.failed);
    if (E > 0) {
        neighbours_kernel<<<blocks((long long)C * 32), kTPB, 0, st>>>(cellKey, C, D, T.key, T.mask, slotCell,
                                                                      nullptr, nbStart, nbList, nbOwner);
        note_launch();
        pair_kernel<<<blocks(E), kTPB, 0, st>>>(K, nbOwner, nbList, eps, pst, openList, joinList, active, openE,
                                                settledE, deferred, counts);
        note_launch();
        rep_pairs_kernel<<<loop, kTPB, 0, st>>>(K, nbOwner, nbList, openList, eps, pst, joinList, counts);
        note_launch();
        if (C <= kSharedCells) {
            const size_t shm = (size_t)C * sizeof(int);
            if (shm > 48 * 1024)
                CK(cudaFuncSetAttribute(cell_components_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
            cell_components_kernel<<<1, 1024, shm, st>>>(C, nbOwner, nbList, joinList, counts + kJoinedCount, parentC);
        } else {
            join_all_kernel<<<blocks(E), kTPB, 0, st>>>(nbOwner, nbList, joinList, counts + kJoinedCount, parentC);
        }
        note_launch();
        CKL();
    }
    // first sort: the points of the cells that are not dense
    const size_t n1 = (size_t)n + 1;
    Sorted Q;
    Q.order = A.take<int>(n1);
    Q.cell = A.take<int>(n1);
    Q.core = A.take<unsigned char>(n1);
    Q.fix = compat ? A.take<unsigned char>(n1) : nullptr;
    for (int d = 0; d < 3; ++d) {
        Q.s[d] = d < D ? A.take<double>(n1) : nullptr;
        Q.r[d] = nullptr;
    }
    Q.sb = K.sb;
    Q.se = K.se;
    Q.D = D;
    ScanQueue W;
    W.cap = (int)std::min<long long>(std::max<long long>(4096, n), 1 << 20);
    W.point = A.take<int>(W.cap);
    W.cell = A.take<int>(W.cap);
    W.count = counts + kScanA;
    const long long words = (n + 31) / 32;
    unsigned* bits = A.take<unsigned>(2 * words);
    int* ranks = A.take<int>(2 * words);
    NEED(!c.failed);
    auto sort_phase = [&](const int* before, int* total) -> int {
        int r = device_scan(c, take, cursor, C, total);
        if (r) return r;
        phase_begin_kernel<<<blocks(C), kTPB, 0, st>>>(C, cursor, take, before, begin, K.sb, K.se, K.cnt);
        note_launch();
        sort_kernel<Src><<<blocks(n), kTPB, 0, st>>>(S, n, slot, slotCell, begin, cursor, Q, K.dense,
                                                     compat ? 1 : 0, total);
        note_launch();
        CKL();
        return CHAOS_OK;
    };
    take_sparse_kernel<<<blocks(C), kTPB, 0, st>>>(K, take);
    note_launch();
    if ((rc = sort_phase(nullptr, counts + kSparse))) return rc;
    // core flags and the shortcuts' links of the points that are not in dense cells
    if (!compat) {
        core_kernel<<<loop, kTPB, 0, st>>>(Q, K, nbStart, nbList, eps, minPts, 0, ScanQueue{}, nullptr, counts);
        note_launch();
    }
    dense_links_kernel<<<loop, kTPB, 0, st>>>(Q, K, nbStart, nbList, eps, parentC, openE, settledE, counts);
    note_launch();
    if (E > 0) {
        open_pairs_kernel<<<blocks(E), kTPB, 0, st>>>(K, nbOwner, nbList, parentC, pst, openE, settledE, active, counts);
        note_launch();
    }
    CKL();
    // second sort: the cells some pair, count or label still has to scan
    take_needed_kernel<<<blocks(C), kTPB, 0, st>>>(K, take);
    note_launch();
    if ((rc = sort_phase(counts + kSparse, counts + kNeeded))) return rc;
    // what is kept per sorted point: its offsets, what the long scans find (a
    // count, later the best component's key) and its nodes. By the points while
    // there are few, otherwise by the number that was sorted, which takes a wait.
    long long M = n;
    if (n > kRoomySet) {
        int hm[kNeeded + 1];
        CK(cudaMemcpyAsync(hm, counts, sizeof hm, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        M = (long long)hm[kSparse] + hm[kNeeded];
    }
    const size_t M1 = (size_t)M + 1, N = (size_t)C + M1;  // nodes: the cells, then the sorted points
    for (int d = 0; d < D; ++d) Q.r[d] = A.take<float>(M1);
    unsigned long long* found = A.take<unsigned long long>(M1);
    int* parent = A.take<int>(N);
    int* compMin = A.take<int>(N);
    int* compFix = A.take<int>(N);
    int* compLabel = A.take<int>(N);
    NEED(!c.failed);
    nodes_kernel<<<loop, kTPB, 0, st>>>(Q, K, parentC, parent, compMin, compFix, counts);
    note_launch();
    if (!compat) {  // the undecided counts, exactly (their neighbours are sorted now)
        core_kernel<<<loop, kTPB, 0, st>>>(Q, K, nbStart, nbList, eps, minPts, 1, W, (int*)found, counts);
        note_launch();
        long_scan_kernel<<<loop, 256, 0, st>>>(Q, K, W, eps, minPts, 0, (int*)found, nullptr, nullptr, nullptr);
        note_launch();
        core_finish_kernel<<<loop, kTPB, 0, st>>>(Q, K, nbStart, nbList, eps, minPts, (const int*)found, parent, counts);
        note_launch();
    }
    // unions
    if (E > 0) {
        whole_pairs_kernel<<<blocks(E), kTPB, 0, st>>>(K, nbOwner, nbList, pst, parent, counts);
        note_launch();
    }
    unsafe_cell_kernel<<<blocks((long long)C * 32), kTPB, 0, st>>>(Q, K, eps, parent);
    note_launch();
    if (E > 0) {
        // (the open list has been read: its memory serves the long pairs)
        for (int pass = 0; pass < kCrossPasses; ++pass) {
            cross_cell_kernel<<<loop, kTPB, 0, st>>>(Q, K, nbOwner, nbList, eps, parent, pass, deferred, openList,
                                                     counts + kLong, active, counts);
            note_launch();
        }
        long_pairs_kernel<<<loop, 256, 0, st>>>(Q, K, nbOwner, nbList, openList, counts + kLong, eps, parent);
        note_launch();
    }
    CKL();
    // components, numbered
    comp_kernel<<<loop, kTPB, 0, st>>>(Q, K, parent, compMin, compFix, counts);
    note_launch();
    CK(cudaMemsetAsync(bits, 0, 2 * words * sizeof(unsigned), st));
    root_marks_kernel<<<loop, kTPB, 0, st>>>(Q, K, parent, compMin, compFix, compat ? 1 : 0, bits, bits + words, counts);
    note_launch();
    const long long ranked = compat ? 2 * words : words;
    bit_counts_kernel<<<blocks(ranked), kTPB, 0, st>>>(bits, ranks, ranked);
    note_launch();
    if ((rc = device_scan(c, ranks, ranks, words, nullptr))) return rc;
    if (compat && (rc = device_scan(c, ranks + words, ranks + words, words, nullptr))) return rc;
    root_labels_kernel<<<loop, kTPB, 0, st>>>(Q, K, parent, compMin, compFix, compat ? 1 : 0, bits, bits + words, ranks,
                                              ranks + words, compLabel, counts);
    note_launch();
    cell_labels_kernel<<<blocks(C), kTPB, 0, st>>>(K, parent, compLabel, cellLabel);
    note_launch();
    labels_kernel<<<blocks(n), kTPB, 0, st>>>(slot, slotCell, n, K.dense, cellLabel, compat ? 1 : 0, labels);
    note_launch();
    W.count = counts + kScanB;
    sorted_labels_kernel<<<loop, kTPB, 0, st>>>(Q, K, nbStart, nbList, eps, parent, compMin, compLabel, labels, W, found,
                                                counts);
    note_launch();
    long_scan_kernel<<<loop, 256, 0, st>>>(Q, K, W, eps, minPts, 1, nullptr, found, parent, compMin);
    note_launch();
    border_labels_kernel<<<loop, kTPB, 0, st>>>(Q, found, compLabel, labels, counts);
    note_launch();
    CKL();
    return CHAOS_OK;
}

}  // namespace

// Exclusive prefix sums; dTotal (device memory, may be null) receives the total.
template <class T>
static int device_scan_t(Call& c, const T* in, T* out, long long n, T* dTotal) {
    if (n <= 0) {
        if (dTotal) CK(cudaMemsetAsync(dTotal, 0, sizeof(T), c.stream));
        return CHAOS_OK;
    }
    const long long nb = (n + kScanItems - 1) / kScanItems;
    T* sums = nb == 1 && dTotal ? dTotal : (T*)c.alloc((size_t)nb * sizeof(T));
    if (!sums) return CHAOS_E_NOMEM;
    scan_block_kernel<T><<<(unsigned)nb, 1024, 0, c.stream>>>(in, out, sums, n);
    note_launch();
    CK(cudaGetLastError());
    if (nb > 1) {
        int rc = device_scan_t<T>(c, sums, sums, nb, dTotal);
        if (rc) return rc;
        add_offsets_kernel<T><<<blocks(n), kTPB, 0, c.stream>>>(out, sums, n);
        note_launch();
        CK(cudaGetLastError());
    }
    return CHAOS_OK;
}

int device_scan(Call& c, const int* in, int* out, long long n, int* dTotal) {
    return device_scan_t<int>(c, in, out, n, dTotal);
}

template <class T>
static int exclusive_scan_t(Call& c, const T* in, T* out, long long n, T* total) {
    T* d = total ? (T*)c.alloc(sizeof(T)) : nullptr;
    if (total && !d) return CHAOS_E_NOMEM;
    int rc = device_scan_t<T>(c, in, out, n, d);
    if (rc || !total) return rc;
    CK(cudaMemcpyAsync(total, d, sizeof(T), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    return CHAOS_OK;
}

int exclusive_scan64(Call& c, const long long* in, long long* out, long long n, long long* total) {
    return exclusive_scan_t<long long>(c, in, out, n, total);
}

int dbscan_compat_device(Call& c, const double* avgPeaks, const double* avgIntervals, const int* flags, long long n,
                         double eps, int* labels) {
    ColSrc S;
    S.f[0] = avgPeaks;
    S.f[1] = avgIntervals;
    S.f[2] = avgIntervals;
    S.mask = nullptr;
    S.flags = flags;
    S.D = 2;
    S.compat = true;
    return cell_cluster(c, S, n, eps, 1, true, 0.0, nullptr, labels);
}

int dbscan_device(Call& c, const double* features, long long n, int dims, double eps, int minPts, const int* mask,
                  int* labels) {
    RowSrc S;
    S.F = features;
    S.mask = mask;
    S.D = dims;
    return cell_cluster(c, S, n, eps, minPts, false, 0.0, nullptr, labels);
}

int dbscan_basins_device(Call& c, const BasinsOut& O, long long n, const unsigned long long* minmaxKeys, double eps,
                         int minPts, double* features, int* labels) {
    BasinSrc S;
    S.flags = O.flags;
    S.counts = O.counts;
    S.avgPeaks = O.avgPeaks;
    S.avgIntervals = O.avgIntervals;
    S.last = O.last;
    S.D = 3;
    for (int d = 0; d < 3; ++d) {
        const bool any = minmaxKeys[d] != ~0ull;
        auto unk = [](unsigned long long k) {
            const unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
            double v;
            memcpy(&v, &b, sizeof v);
            return v;
        };
        const double lo = any ? unk(minmaxKeys[d]) : 0.0, hi = any ? unk(minmaxKeys[3 + d]) : 0.0;
        S.lo[d] = lo;
        S.ok[d] = any && hi > lo;
        S.inv[d] = S.ok[d] ? 1.0 / (hi - lo) : 0.0;
    }
    // normalised features lie in [0, 1]: at most floor(1 / side) + 1 cells per
    // dimension (one more for the rounding of (f - lo) * inv), and one cell
    // of NaN features
    const double side = eps / sqrt(3.0) * (1.0 - 1e-9);
    const double per = floor(1.0 / side) + 2.0;
    const double bound = per * per * per + 1.0;
    return cell_cluster(c, S, n, eps, minPts, false, bound, features, labels);
}

}  // namespace chaos
