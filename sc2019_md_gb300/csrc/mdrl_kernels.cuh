/*
 * mdrl_kernels.cuh — sm_103a kernels of the range-limited force path.
 *
 * Data layout in HBM (all particle arrays are in cell-sorted order after binning):
 *   pos   float4[n]  (x, y, z, q)        one 16-byte coalesced load per particle
 *   type  int[n]
 *   F     3 x int64[n] (SoA, 2^-24 kcal/mol/A fixed point) or 3 x float[n] (FP32-atomic mode)
 *   cell_start int[ncells + 1]           cell c holds sorted particles [start[c], start[c+1])
 *
 * Pair datapath, per candidate (the reference RTL order, SC/r2_compute_with_pbc.v:81-127,
 * SC/Filter_Logic.v:234, SC/RL_LJ_Evaluate_Pairs_1st_Order.v:179-193,409-468,
 * SC/RL_Evaluate_Pairs_1st_Order.v:325-395):
 *   d = x_ref - x_nbr, one conditional +-L wrap per axis;
 *   r2 = (dx*dx + dy*dy) + dz*dz, each operation rounded (the pair list is bit-identical to an
 *        all-pairs FP32 evaluation of the same positions);
 *   keep when 0 < r2 <= rc2;
 *   table index = (exponent(r2) - 127 - min_log2) * bins + top mantissa bits;
 *   v_k = c1*r2 + c0 (or Horner for orders 2-3), fscal = ((QQ*v3) + B*v8) + A*v14,
 *   f = fscal * d, added to i and subtracted from j (Newton's third law).
 */
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mdrl_internal.h"

namespace mdrl {

/* Tables packed for the kernels: for order 1, per table index three float2 {c0, c1} (force:
 * r^-14, r^-8, r^-3; energy: r^-12, r^-6, r^-1); for orders 2-3, three float4 {c0..c3}.
 * Polynomial form: monomial in r2 (the reference's form: c0 + c1 r2 + ...), or, when `local`
 * is set (orders 2-3), in the bin-local variable u = r2 - b0, b0 the start of r2's bin.  u is
 * exact in FP32 (r2 and b0 share a binade and b0 <= r2 < 2 b0), so the local form carries no
 * cancellation between large monomial terms. */
struct TableDev {
    const float2 *f2, *e2;
    const float4 *f4, *e4;
    const float4 *fr;   /* order 1, force functions packed per index in one 32-byte sector:
                           {c0_14, c1_14, c0_8, c1_8}, {c0_3, c1_3, 0, 0} */
    /* the one-warp-per-item and list kernels' copies of the force functions, split so that a gather's lanes spread over
     * every 16-byte bank group: order 1 wa {c0_14, c1_14, c0_8, c1_8}, wc {c0_3, c1_3}; order 2 wa
     * {c0_14, c1_14, c2_14, c0_8}, wb {c1_8, c2_8, c0_3, c1_3}, w1 c2_3 */
    const float4 *wa, *wb;
    const float2 *wc;
    const float *w1;
    int order, nseg, bins, lb, min_log2;
    float r2min;
    int local;          /* orders 2-3: coefficients in u = r2 - bin start */
    unsigned bmask;     /* local: the r2 bits that give the bin start; else 0 (u = r2) */
};

/* The polynomial variable of an in-table r2e: r2e itself, or r2e minus its bin's start (the r2
 * bit pattern with the mantissa bits below the bin index cleared). */
__device__ __forceinline__ float table_variable(const TableDev &t, float r2e) {
    if (!t.local) return r2e;
    const float b0 = __uint_as_float(__float_as_uint(r2e) & ~((1u << (23 - t.lb)) - 1u));
    return __fsub_rn(r2e, b0);
}

/* The 14 cells of the half shell in the reference's filter order (mdrl_internal.h). */
__constant__ int c_halfshell[kHalfShellCells][3] = MDRL_HALFSHELL_OFFSETS;

/* Error bits raised by kernels and read by the host after a call.  kErrForce: a force sum that
 * the accumulators cannot hold -- NaN or infinite, or (int64 fixed point) a magnitude at or above
 * kFixMax, which the conversion would saturate. */
enum : unsigned { kErrPosition = 1u, kErrType = 2u, kErrForce = 4u, kErrCellOverflow = 8u };

/* Cell occupancy: cells up to kSortSmall particles are ordered in one shared-memory pass; larger
 * ones in sorted chunks of kSortSmall merged by binary search; above kMaxCellOcc a cell raises
 * kErrCellOverflow (MDRL_ERR_CELL_OVERFLOW), keeps its arrival order, and the force kernel skips
 * the units that touch it, so a pathological input costs bounded time. */
constexpr int kSortSmall = 1024;
constexpr int kMaxCellOcc = 65536;

/* The largest force (kcal/mol/A) a 2^-24 fixed-point component holds without saturating: the
 * conversion clamps at 9e18 units. */
constexpr float kFixMax = 9.0e18f / 16777216.0f;

/* Per-type mass factors, kept in device memory and read through a pointer (a by-value kernel
 * parameter indexed by a particle's type would be copied to local memory in every thread). */
struct MassTab {
    float cm[MDRL_MAX_TYPES];   /* velocity increment per unit force for the kick */
    float mass[MDRL_MAX_TYPES]; /* amu, for the kinetic energy */
};

__device__ __forceinline__ float wrap_d(float d, float L, float h) {
    return d > h ? __fsub_rn(d, L) : (d < -h ? __fadd_rn(d, L) : d);
}

/* The exact-difference rule per pair (MDRL_FLAG_EXACT_DIFF): the wrap direction from fl(xi - xj)
 * as above, then the box edge comes off the high coordinate (exact for coordinates in [0, L):
 * the one wrapped lies above L/2) and the difference is rounded once. */
__device__ __forceinline__ float wrap_exact(float xi, float xj, float L, float h) {
    const float d = __fsub_rn(xi, xj);
    if (d > h) return __fsub_rn(__fsub_rn(xi, L), xj);
    if (d < -h) return __fsub_rn(xi, __fsub_rn(xj, L));
    return d;
}

/* s + e = a + b exactly (Knuth's two-sum) */
__device__ __forceinline__ float two_sum(float a, float b, float &e) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return s;
}

template <bool SEP>
__device__ __forceinline__ float madd(float a, float b, float c) {
    return SEP ? __fadd_rn(__fmul_rn(a, b), c) : __fmaf_rn(a, b, c);
}

__device__ __forceinline__ int table_index(const TableDev &t, float r2, float &r2e, int &below) {
    const unsigned b = __float_as_uint(r2);
    int seg = (int)(b >> 23) - 127 - t.min_log2;
    int bin = (int)((b >> (23 - t.lb)) & (unsigned)(t.bins - 1));
    r2e = r2;
    below = 0;
    if (seg < 0) {
        seg = 0; bin = 0; r2e = t.r2min; below = 1;
    } else if (seg >= t.nseg) {
        seg = t.nseg - 1; bin = t.bins - 1;
    }
    return seg * t.bins + bin;
}

template <int ORDER, bool SEP>
__device__ __forceinline__ float poly4(float4 c, float x) {
    float v = (ORDER >= 3) ? c.w : c.z;
    if (ORDER >= 3) v = madd<SEP>(v, x, c.z);
    v = madd<SEP>(v, x, c.y);
    return madd<SEP>(v, x, c.x);
}

/* The pair functions v14, v8, v3 (and v12, v6, v1 when ENERGY) at r2. */
template <int ORDER, bool SEP, bool ENERGY>
__device__ __forceinline__ void pair_functions(const TableDev &t, float r2, bool coul, float &v14,
                                               float &v8, float &v3, float &v12, float &v6,
                                               float &v1, int &below) {
    if (ORDER == 0) {
        const float i2 = __fdiv_rn(1.0f, r2);
        const float i4 = __fmul_rn(i2, i2), i6 = __fmul_rn(i4, i2), i8 = __fmul_rn(i4, i4);
        const float i12 = __fmul_rn(i6, i6), i14 = __fmul_rn(i12, i2);
        const float i1 = __fsqrt_rn(i2), i3 = __fmul_rn(i2, i1);
        v14 = i14; v8 = i8; v3 = i3; v12 = i12; v6 = i6; v1 = i1;
        below = 0;
        return;
    }
    float r2e;
    const int idx = table_index(t, r2, r2e, below);
    if (ORDER == 1) {
        const float2 a = __ldg(t.f2 + 3 * idx), b = __ldg(t.f2 + 3 * idx + 1);
        v14 = madd<SEP>(a.y, r2e, a.x);
        v8 = madd<SEP>(b.y, r2e, b.x);
        v3 = 0.0f;
        if (coul) { const float2 c = __ldg(t.f2 + 3 * idx + 2); v3 = madd<SEP>(c.y, r2e, c.x); }
        if (ENERGY) {
            const float2 d = __ldg(t.e2 + 3 * idx), e = __ldg(t.e2 + 3 * idx + 1);
            v12 = madd<SEP>(d.y, r2e, d.x);
            v6 = madd<SEP>(e.y, r2e, e.x);
            v1 = 0.0f;
            if (coul) { const float2 g = __ldg(t.e2 + 3 * idx + 2); v1 = madd<SEP>(g.y, r2e, g.x); }
        }
    } else {
        const float x = table_variable(t, r2e);
        v14 = poly4<ORDER, SEP>(__ldg(t.f4 + 3 * idx), x);
        v8 = poly4<ORDER, SEP>(__ldg(t.f4 + 3 * idx + 1), x);
        v3 = coul ? poly4<ORDER, SEP>(__ldg(t.f4 + 3 * idx + 2), x) : 0.0f;
        if (ENERGY) {
            v12 = poly4<ORDER, SEP>(__ldg(t.e4 + 3 * idx), x);
            v6 = poly4<ORDER, SEP>(__ldg(t.e4 + 3 * idx + 1), x);
            v1 = coul ? poly4<ORDER, SEP>(__ldg(t.e4 + 3 * idx + 2), x) : 0.0f;
        }
    }
}

/* fscal = ((QQ*v3) + B*v8) + A*v14 ; energies el = Be*v6 + Ae*v12, ec = QQ*v1. */
template <bool SEP>
__device__ __forceinline__ float combine_force(float4 pc, float qq, bool coul, float v14, float v8,
                                               float v3) {
    if (SEP) {
        float fs = __fmul_rn(pc.y, v8);
        if (coul) fs = __fadd_rn(__fmul_rn(qq, v3), fs);
        return __fadd_rn(fs, __fmul_rn(pc.x, v14));
    }
    const float fs = __fmaf_rn(pc.y, v8, coul ? __fmul_rn(qq, v3) : 0.0f);
    return __fmaf_rn(pc.x, v14, fs);
}

template <bool SEP>
__device__ __forceinline__ float combine_elj(float4 pc, float v12, float v6) {
    return SEP ? __fadd_rn(__fmul_rn(pc.w, v6), __fmul_rn(pc.z, v12))
               : __fmaf_rn(pc.z, v12, __fmul_rn(pc.w, v6));
}

/* 2^-24 fixed point.  NaN converts to 0 and magnitudes beyond kFixMax saturate; callers report
 * both through force_ok / kErrForce rather than let them pass silently. */
__device__ __forceinline__ unsigned long long to_fixed(float v) {
    float s = v * kFixScale;
    if (!(s == s)) s = 0.0f;
    s = fminf(fmaxf(s, -9.0e18f), 9.0e18f);
    return (unsigned long long)__float2ll_rn(s);
}

/* True when every component is finite and below kFixMax in magnitude (NaN fails the compare). */
__device__ __forceinline__ bool force_ok(float fx, float fy, float fz) {
    return fabsf(fx) < kFixMax && fabsf(fy) < kFixMax && fabsf(fz) < kFixMax;
}

/* Raise kErrForce when a force sum cannot be represented (one atomic per offending thread). */
__device__ __forceinline__ void check_force(unsigned *err, float fx, float fy, float fz) {
    if (!force_ok(fx, fy, fz) && err) atomicOr(err, kErrForce);
}

__device__ __forceinline__ float from_fixed(unsigned long long v) {
    return __ll2float_rn((long long)v) * kFixInv;
}

/* ------------------------------------------------------------------------------------------ */
/* Binning: cell = floor(pos / edge) (MS/GenInputCellList_LJArgon.m:98-112), stable within the
 * cell (input order, :114-121).  count -> scan -> scatter -> per-cell rank sort.              */

__device__ __forceinline__ int cell_coord(float v, float edge, int n) {
    const float f = floorf(__fdiv_rn(v, edge));
    if (!(f >= 0.0f)) return 0;
    if (f >= (float)n) return n - 1;
    return (int)f;
}

__device__ __forceinline__ int cell_of_pos(const Geom &g, float x, float y, float z) {
    const int cx = cell_coord(x, g.edge[0], g.nc[0]);
    const int cy = cell_coord(y, g.edge[1], g.nc[1]);
    const int cz = cell_coord(z, g.edge[2], g.nc[2]);
    return (cx * g.nc[1] + cy) * g.nc[2] + cz;
}

/* 30-bit Morton code of a position inside its cell (10 bits per axis): the in-cell sort key of
 * the force path.  Only an ordering, so its rounding does not matter; ties break on the index. */
__device__ __forceinline__ unsigned spread10(unsigned v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__device__ __forceinline__ unsigned cell_morton(const Geom &g, float x, float y, float z, int c) {
    const int cz = c % g.nc[2], cy = (c / g.nc[2]) % g.nc[1], cx = c / (g.nc[1] * g.nc[2]);
    const float p[3] = {x, y, z};
    const int cc[3] = {cx, cy, cz};
    unsigned q[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        /* an ordering only: the fast reciprocal (deterministic) is as good as an IEEE division */
        const float loc = (p[d] - (float)cc[d] * g.edge[d]) * __fdividef(1024.0f, g.edge[d]);
        q[d] = (unsigned)min(1023, max(0, (int)loc));
    }
    return (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
}

/* The in-cell sort key of the list kernel: the position's index on a 3-D Hilbert curve through the
 * cell, 8 bits per axis.  Only an ordering, so its rounding does not matter; ties break on the
 * particle index.  Runs of a Hilbert curve are connected, so the 4-, 8- and 32-particle runs that
 * the force kernels box are more compact than those of a Morton curve, which jumps between octants
 * (92k system: 20.7 instead of 23.0 candidate rows of 32 per particle left after culling). */
__device__ __forceinline__ unsigned spread8(unsigned v) {
    v = (v | (v << 8)) & 0x0000f00fu;
    v = (v | (v << 4)) & 0x000c30c3u;
    v = (v | (v << 2)) & 0x00249249u;
    return v;
}

/* Coordinates to the index along the curve: J. Skilling, "Programming the Hilbert curve", AIP Conf.
 * Proc. 707 (2004) 381: undo the excess rotations bit by bit from the top, Gray encode, interleave. */
__device__ __forceinline__ unsigned hilbert24(unsigned x, unsigned y, unsigned z) {
#pragma unroll
    for (unsigned bit = 128u; bit > 1u; bit >>= 1) {
        const unsigned low = bit - 1u;
        if (x & bit) x ^= low;
        unsigned t = (y & bit) ? 0u : ((x ^ y) & low);
        x ^= (y & bit) ? low : t;
        y ^= t;
        t = (z & bit) ? 0u : ((x ^ z) & low);
        x ^= (z & bit) ? low : t;
        z ^= t;
    }
    y ^= x;
    z ^= y;
    unsigned t = 0u;
#pragma unroll
    for (unsigned bit = 128u; bit > 1u; bit >>= 1)
        if (z & bit) t ^= bit - 1u;
    return (spread8(x ^ t) << 2) | (spread8(y ^ t) << 1) | spread8(z ^ t);
}

__device__ __forceinline__ unsigned cell_hilbert(const Geom &g, float x, float y, float z, int c) {
    const int cz = c % g.nc[2], cy = (c / g.nc[2]) % g.nc[1], cx = c / (g.nc[1] * g.nc[2]);
    const float p[3] = {x, y, z};
    const int cc[3] = {cx, cy, cz};
    unsigned q[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        /* an ordering only: the fast reciprocal (deterministic) is as good as an IEEE division */
        const float loc = (p[d] - (float)cc[d] * g.edge[d]) * __fdividef(256.0f, g.edge[d]);
        q[d] = (unsigned)min(255, max(0, (int)loc));
    }
    return hilbert24(q[0], q[1], q[2]);
}

__device__ __forceinline__ bool in_box(const Geom &g, float x, float y, float z) {
    return x >= 0.0f && x < g.L[0] && y >= 0.0f && y < g.L[1] && z >= 0.0f && z < g.L[2];
}

/* Arrival slot of a particle in cell c: lanes of a warp that share c take consecutive slots with
 * one atomic per distinct cell (cell-sorted particles mostly share cells within a warp). */
__device__ __forceinline__ int cell_slot(int *count, int c) {
    const unsigned active = __activemask();
    const unsigned peers = __match_any_sync(active, c);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int base = 0;
    if (lane == leader) base = atomicAdd(count + c, __popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + rank;
}

/* Cell of each user-order particle, with its arrival slot in the cell.  With ux non-null the
 * user arrays (which may be pinned host memory read over the host link) are also copied, in
 * coalesced order, to device staging ux, uy, uz, uq (q given), ut (type given), so that the
 * gather that follows reads device memory. */
static __global__ void k_bin_user(int n, const float *__restrict__ x, const float *__restrict__ y,
                           const float *__restrict__ z, Geom g, int *__restrict__ cell_of,
                           int *__restrict__ slot, int *__restrict__ count,
                           unsigned *__restrict__ err, unsigned *__restrict__ key,
                           const float *__restrict__ q = nullptr, const int *__restrict__ type = nullptr,
                           float *__restrict__ ux = nullptr, float *__restrict__ uy = nullptr,
                           float *__restrict__ uz = nullptr, float *__restrict__ uq = nullptr,
                           int *__restrict__ ut = nullptr, int hilbert = 0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float px = x[i], py = y[i], pz = z[i];
    if (ux) {
        ux[i] = px; uy[i] = py; uz[i] = pz;
        if (q) uq[i] = q[i];
        if (type) ut[i] = type[i];
    }
    if (!in_box(g, px, py, pz)) atomicOr(err, kErrPosition);
    const int c = cell_of_pos(g, px, py, pz);
    cell_of[i] = c;
    if (key) key[i] = hilbert ? cell_hilbert(g, px, py, pz, c) : cell_morton(g, px, py, pz, c);
    slot[i] = cell_slot(count, c);
}

/* The list kernel's tiles: a cell's groups of 4 particles are cut into tiles of at most `groups` groups,
 * the low byte of it for the column classes 0 and 1, the next for class 2.  The scan of the counts numbers
 * them, start[p] the first tiles of cell p (x, y: the two kinds), and the in-cell sort writes tile[kind][k] =
 * (cell, tile of the cell).  So a launch has one item per tile that there is, however unevenly the cells
 * are filled.  Batches: pos[c] the place of cell c in the order of the scan (-1: none), groups by cell. */
struct Tiles {
    int groups = 0;
    int2 *start = nullptr;       /* null: no tiles wanted */
    int2 *tile[2] = {nullptr, nullptr};
    const int *pos = nullptr, *cell_groups = nullptr;
};

/* Tiles of 4 or 8 groups of a cell of m particles (none above the occupancy limit: what touches the cell
 * is skipped). */
__host__ __device__ constexpr int cell_tiles(int m, int groups) {
    return m > kMaxCellOcc ? 0 : (groups == 8 ? (m + 31) >> 5 : (m + 15) >> 4);
}
__device__ __forceinline__ unsigned long long cell_tiles2(int m, int groups) {
    return ((unsigned long long)cell_tiles(m, groups >> 8) << 32) | (unsigned)cell_tiles(m, groups & 0xff);
}
__device__ __forceinline__ int2 tiles_of(unsigned long long v) { return make_int2((int)(unsigned)v, (int)(v >> 32)); }

/* The sum of `own` over the threads before this one plus carry; carry grows by the CTA's sum (1,024
 * threads, one barrier: s_sum is another one at the next call). */
template <class T>
__device__ __forceinline__ T block_scan(T own, T &carry, T (&s_sum)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T sum = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    if (lane == 31) s_sum[warp] = sum;
    __syncthreads();
    T ws = s_sum[lane];                  /* every warp scans the warp sums for itself */
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T v = __shfl_up_sync(0xffffffffu, ws, o);
        if (lane >= o) ws += v;
    }
    const T before = __shfl_sync(0xffffffffu, ws, max(warp - 1, 0));
    const T first = carry + (warp ? before : T(0)) + sum - own;
    carry += __shfl_sync(0xffffffffu, ws, 31);
    return first;
}

/* Exclusive scan of the cell counts (one CTA), plus the largest occupancy, and of the tiles if wanted; zeroes the totals' counts and
 * the force launches' item counters work[0..1] on the way (a memset less per launch), and with clear the
 * counts it has read, for the next step's binning.  Latency-bound: 4 counts per
 * thread and pass in one 16-byte load, warp scans by shuffles, one barrier per pass of 4,096 cells.
 * (A strided run of cells per thread and a 20-barrier scan: 486 cells 3.8 us, 10,648 cells 9.9 us, 28k
 * cells 53 us; now 2.2, 3.3 and 6.) */
static __global__ void __launch_bounds__(1024) k_scan(int ncells, int *__restrict__ count, int *__restrict__ start,
                                               DevTotals *tot, int *work = nullptr, bool clear = false,
                                               Tiles tl = Tiles()) {
    __shared__ int s_sum[2][32], s_max[32];
    __shared__ unsigned long long s_tiles[2][32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned long long tcarry = 0ull;
    if (work && t < 2) work[t] = 0;
    if (t == 0) tot->pairs = tot->below = 0ull;
    int carry = 0, mx = 0, pass = 0;
    for (int base = 0; base < ncells; base += 4096, pass ^= 1) {
        const int k = base + 4 * t;
        int4 c = make_int4(0, 0, 0, 0);
        if (k + 3 < ncells) c = *reinterpret_cast<const int4 *>(count + k);
        else {
            if (k < ncells) c.x = count[k];
            if (k + 1 < ncells) c.y = count[k + 1];
            if (k + 2 < ncells) c.z = count[k + 2];
        }
        if (clear) {
            if (k + 3 < ncells) *reinterpret_cast<int4 *>(count + k) = make_int4(0, 0, 0, 0);
            else
                for (int u = k; u < ncells; ++u) count[u] = 0;
        }
        mx = max(mx, max(max(c.x, c.y), max(c.z, c.w)));
        const int first = block_scan(c.x + c.y + c.z + c.w, carry, s_sum[pass]);
        if (tl.start) {
            const unsigned long long t0 = cell_tiles2(c.x, tl.groups), t1 = t0 + cell_tiles2(c.y, tl.groups),
                                     t2 = t1 + cell_tiles2(c.z, tl.groups), t3 = t2 + cell_tiles2(c.w, tl.groups);
            const unsigned long long f = block_scan(t3, tcarry, s_tiles[pass]);
            const int2 a = tiles_of(f), b = tiles_of(f + t0), d = tiles_of(f + t1), e = tiles_of(f + t2);
            if (k + 3 < ncells) {
                *reinterpret_cast<int4 *>(tl.start + k) = make_int4(a.x, a.y, b.x, b.y);
                *reinterpret_cast<int4 *>(tl.start + k + 2) = make_int4(d.x, d.y, e.x, e.y);
            } else {
                if (k < ncells) tl.start[k] = a;
                if (k + 1 < ncells) tl.start[k + 1] = b;
                if (k + 2 < ncells) tl.start[k + 2] = d;
            }
        }
        const int4 r = make_int4(first, first + c.x, first + c.x + c.y, first + c.x + c.y + c.z);
        if (k + 3 < ncells) *reinterpret_cast<int4 *>(start + k) = r;
        else {
            if (k < ncells) start[k] = r.x;
            if (k + 1 < ncells) start[k + 1] = r.y;
            if (k + 2 < ncells) start[k + 2] = r.z;
        }
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) s_max[warp] = mx;
    __syncthreads();
    if (warp == 0) {
        mx = __reduce_max_sync(0xffffffffu, s_max[lane]);
        if (lane == 0) {
            start[ncells] = carry;
            tot->max_occ = mx;
            if (tl.start) tl.start[ncells] = tiles_of(tcarry);
        }
    }
}

/* The tiles of a batch's cells in another order than the storage's: place p holds cell cell_at[p]. */
static __global__ void __launch_bounds__(1024) k_tile_scan(int nplaces, const int *__restrict__ cell_at,
                                                    const int *__restrict__ count, Tiles tl) {
    __shared__ unsigned long long s_tiles[2][32];
    unsigned long long carry = 0ull;
    int pass = 0;
    for (int base = 0; base < nplaces; base += 4096, pass ^= 1) {
        const int p = base + 4 * threadIdx.x;
        unsigned long long t[4], sum = 0ull;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = p + u < nplaces ? cell_at[p + u] : -1;
            t[u] = sum;
            if (c >= 0) sum += cell_tiles2(count[c], tl.cell_groups[c]);
        }
        const unsigned long long f = block_scan(sum, carry, s_tiles[pass]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (p + u < nplaces) tl.start[p + u] = tiles_of(f + t[u]);
    }
    if (threadIdx.x == 0) tl.start[nplaces] = tiles_of(carry);
}

static __global__ void k_scatter(int n, const int *__restrict__ cell_of, const int *__restrict__ slot,
                          const int *__restrict__ start, int *__restrict__ tmp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    tmp[start[cell_of[i]] + slot[i]] = i;
}

/* Also writes the cells' tiles (tl).  Order each cell's particles: by index (the reference's in-cell order, input order), or, when
 * key is given, by (key, index).  The rank of an element is the number of smaller ones (the
 * (key, index) pairs are distinct).  scratch[n] (64-bit) holds the sorted chunks of cells above
 * kSortSmall. */
static __global__ void __launch_bounds__(128) k_cell_sort(const int *__restrict__ start,
                                                          const int *__restrict__ tmp,
                                                          int *__restrict__ sorted,
                                                          const unsigned *__restrict__ key,
                                                          unsigned long long *__restrict__ scratch,
                                                          unsigned *__restrict__ err, Tiles tl = Tiles()) {
    __shared__ __align__(16) unsigned long long s_k[kSortSmall];
    const int c = blockIdx.x;
    const int s = start[c], m = start[c + 1] - s;
    if (m == 0) return;
    const int place = !tl.start ? -1 : (tl.pos ? tl.pos[c] : c);
    if (place >= 0) {
        const int g = tl.cell_groups ? tl.cell_groups[c] : tl.groups;
        const int2 at = tl.start[place];
        for (int t = threadIdx.x; t < cell_tiles(m, g & 0xff); t += blockDim.x) tl.tile[0][at.x + t] = make_int2(c, t);
        for (int t = threadIdx.x; t < cell_tiles(m, g >> 8); t += blockDim.x) tl.tile[1][at.y + t] = make_int2(c, t);
    }
    if (m > kMaxCellOcc) {
        if (threadIdx.x == 0) atomicOr(err, kErrCellOverflow);
        for (int e = threadIdx.x; e < m; e += blockDim.x) sorted[s + e] = tmp[s + e];
        return;
    }
    if (m <= kSortSmall) {
        for (int e = threadIdx.x; e < m; e += blockDim.x) {
            const int id = tmp[s + e];
            s_k[e] = ((unsigned long long)(key ? key[id] : 0u) << 32) | (unsigned)id;
        }
        if ((m & 1) && threadIdx.x == 0) s_k[m] = ~0ull;     /* pad to an even count: never smaller */
        __syncthreads();
        const int m2 = (m + 1) >> 1;
        const ulonglong2 *s_k2 = reinterpret_cast<const ulonglong2 *>(s_k);
        for (int e = threadIdx.x; e < m; e += blockDim.x) {
            const unsigned long long me = s_k[e];
            /* rank = number of smaller keys; two keys per shared load, four independent counters */
            int r0 = 0, r1 = 0, r2 = 0, r3 = 0;
            int q = 0;
            for (; q + 1 < m2; q += 2) {
                const ulonglong2 a = s_k2[q], b = s_k2[q + 1];
                r0 += a.x < me; r1 += a.y < me; r2 += b.x < me; r3 += b.y < me;
            }
            if (q < m2) { const ulonglong2 a = s_k2[q]; r0 += a.x < me; r1 += a.y < me; }
            sorted[s + r0 + r1 + r2 + r3] = (int)(me & 0xffffffffu);
        }
        return;
    }
    /* large cell: sort each chunk of kSortSmall in shared memory (rank count) into scratch ... */
    for (int c0 = 0; c0 < m; c0 += kSortSmall) {
        const int mc = min(kSortSmall, m - c0);
        __syncthreads();
        for (int e = threadIdx.x; e < mc; e += blockDim.x) {
            const int id = tmp[s + c0 + e];
            s_k[e] = ((unsigned long long)(key ? key[id] : 0u) << 32) | (unsigned)id;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < mc; e += blockDim.x) {
            const unsigned long long me = s_k[e];
            int r = 0;
            for (int q = 0; q < mc; ++q) r += s_k[q] < me;
            scratch[s + c0 + r] = me;
        }
    }
    __syncthreads();   /* the block's global writes are visible to the block after the barrier */
    /* ... then an element's rank = its rank in its chunk + the keys below it in every other chunk
     * (binary search: O(m log kSortSmall / kSortSmall) per element) */
    for (int e = threadIdx.x; e < m; e += blockDim.x) {
        const unsigned long long me = scratch[s + e];
        const int ce = e / kSortSmall;
        int r = e - ce * kSortSmall;
        for (int c0 = 0, cc = 0; c0 < m; c0 += kSortSmall, ++cc) {
            if (cc == ce) continue;
            const unsigned long long *a = scratch + s + c0;
            int lo = 0, hi = min(kSortSmall, m - c0);   /* first index with a[idx] >= me */
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (a[mid] < me) lo = mid + 1; else hi = mid;
            }
            r += lo;
        }
        sorted[s + r] = (int)(me & 0xffffffffu);
    }
}

/* Gather user-order inputs into cell order and clear the force accumulators. */
static __global__ void k_gather_user(int n, const int *__restrict__ sorted, const float *__restrict__ x,
                              const float *__restrict__ y, const float *__restrict__ z,
                              const float *__restrict__ q, const int *__restrict__ type,
                              float4 *__restrict__ pos, int *__restrict__ ptype,
                              int *__restrict__ pid, unsigned long long *__restrict__ F64,
                              float *__restrict__ F32, int *__restrict__ counts, int ntypes,
                              unsigned *__restrict__ err, int *__restrict__ inv = nullptr) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int id = sorted[k];
    if (inv) inv[id] = k;
    pos[k] = make_float4(x[id], y[id], z[id], q ? q[id] : 0.0f);
    int t = type ? type[id] : 0;
    if (t < 0 || t >= ntypes) { atomicOr(err, kErrType); t = 0; }
    ptype[k] = t;
    pid[k] = id;
    if (F64) { F64[k] = 0ull; F64[n + k] = 0ull; F64[2 * n + k] = 0ull; }
    if (F32) {
#pragma unroll
        for (int d = 0; d < 6; ++d) F32[(size_t)d * n + k] = 0.0f;   /* hi planes 0-2, lo planes 3-5 */
    }
    if (counts) counts[k] = 0;
}

/* Totals over units and kinetic-energy partials, in a fixed order: CTA b of nb sums the units and
 * partials of its threads' stride into part[b], and the last CTA to finish sums those.  GB300 runs
 * FP64 at a small fraction of its FP32 rate (2 lanes per SM and cycle), so the sums are spread over
 * SMs and halve the active threads at every level; the FP64 ones run only when energies were computed.
 * (One CTA of 1,024 threads with warp-shuffle sums: 378 units with energies 10.5 us, 6,804 units 7.3 us,
 * 149k units 29 us, the 512-replica batch 142 us; now 3, 3, 4 and 8.) */
constexpr int kTotThreads = 256, kTotBlocks = 128;
struct TotPart {
    double e[4];                     /* LJ, Coulomb, virial, kinetic */
    unsigned long long u[2];         /* pairs, below the table */
};
struct TotScratch {
    TotPart part[kTotBlocks];
    unsigned done;                   /* CTAs finished; 0 between launches */
};
/* The result slots of a force launch: n; or of an evaluation by lists n, then count[0] more and, from slot
 * `second` on, count2[0] (null: none), numbers that the launches have left on the device. */
struct TotUnits {
    int n;
    const int *count = nullptr, *count2 = nullptr;
    int second = 0;
};
inline int tot_blocks(int nunits, int nke) {
    const int b = ((nunits > nke ? nunits : nke) + 4 * kTotThreads - 1) / (4 * kTotThreads);
    return b < 1 ? 1 : (b > kTotBlocks ? kTotBlocks : b);
}

__device__ __forceinline__ void tot_tree(TotPart *s, int n, bool fp) {
    for (int o = kTotThreads / 2; o > 0; o >>= 1) {
        if (o < n && (int)threadIdx.x < o) {     /* entries from n on are zero */
            TotPart &a = s[threadIdx.x];
            const TotPart &b = s[threadIdx.x + o];
            if (fp) {
#pragma unroll
                for (int k = 0; k < 4; ++k) a.e[k] += b.e[k];
            }
            a.u[0] += b.u[0];
            a.u[1] += b.u[1];
        }
        __syncthreads();
    }
}

static __global__ void __launch_bounds__(kTotThreads) k_totals(TotUnits units, const UnitOut *__restrict__ uout,
                                                               int nke, const double *__restrict__ kepart,
                                                               DevTotals *tot, int with_energy, TotScratch *scr) {
    const int upto = units.n + (units.count ? units.count[0] : 0);      /* slots [0, upto), then those from second */
    const int nunits = upto + (units.count2 ? units.count2[0] : 0), skip = units.second - upto;
    __shared__ TotPart s[kTotThreads];
    __shared__ unsigned s_last;
    const int t = threadIdx.x, stride = gridDim.x * kTotThreads;
    const bool fp = with_energy || nke > 0;
    TotPart a{};
#pragma unroll 4
    for (int u = blockIdx.x * kTotThreads + t; u < nunits; u += stride) {
        const UnitOut &o = uout[u < upto ? u : u + skip];
        a.u[0] += o.pairs;
        if (with_energy) {
            a.e[0] += o.e_lj; a.e[1] += o.e_coul; a.e[2] += o.virial;
            a.u[1] += o.below;
        }
    }
#pragma unroll 4
    for (int u = blockIdx.x * kTotThreads + t; u < nke; u += stride) a.e[3] += kepart[u];
    s[t] = a;
    __syncthreads();
    tot_tree(s, min(kTotThreads, (nunits > nke ? nunits : nke) - (int)blockIdx.x * kTotThreads), fp);
    if (gridDim.x > 1) {
        if (t == 0) {
            scr->part[blockIdx.x] = s[0];
            __threadfence();
            s_last = atomicAdd(&scr->done, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        s[t] = t < (int)gridDim.x ? scr->part[t] : TotPart{};
        if (t == 0) scr->done = 0;
        __syncthreads();
        tot_tree(s, gridDim.x, fp);
    }
    if (t == 0) {
        tot->e_lj = s[0].e[0]; tot->e_coul = s[0].e[1]; tot->virial = s[0].e[2];
        tot->e_bond = tot->e_angle = tot->e_dihedral = 0.0;   /* the bonded kernel adds its own */
        if (nke > 0) tot->kinetic = s[0].e[3];
        tot->pairs = s[0].u[0]; tot->below = s[0].u[1];
        tot->pairs_total += s[0].u[0];
    }
}

/* Sorted forces back to user order as float (and counts). */
static __global__ void k_unsort(int n, const int *__restrict__ pid, const unsigned long long *__restrict__ F64,
                         const float *__restrict__ F32, const int *__restrict__ cnt_s,
                         float *__restrict__ fx, float *__restrict__ fy, float *__restrict__ fz,
                         int *__restrict__ cnt_u) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int id = pid[k];
    if (F64) {
        fx[id] = from_fixed(F64[k]); fy[id] = from_fixed(F64[n + k]); fz[id] = from_fixed(F64[2 * n + k]);
    } else {
        fx[id] = F32[k] + F32[3 * (size_t)n + k];
        fy[id] = F32[n + k] + F32[4 * (size_t)n + k];
        fz[id] = F32[2 * n + k] + F32[5 * (size_t)n + k];
    }
    if (cnt_u) cnt_u[id] = cnt_s[k];
}

/* The same in user order (inv = cell-order position of each user index): the writes are
 * coalesced, so fx, fy, fz, cnt_u may be pinned host memory written over the host link. */
static __global__ void k_unsort_inv(int n, const int *__restrict__ inv, const unsigned long long *__restrict__ F64,
                                    const float *__restrict__ F32, const int *__restrict__ cnt_s,
                                    float *__restrict__ fx, float *__restrict__ fy, float *__restrict__ fz,
                                    int *__restrict__ cnt_u, const DevTotals *__restrict__ tot_d = nullptr,
                                    DevTotals *tot_h = nullptr, const unsigned *__restrict__ err_d = nullptr,
                                    unsigned *err_h = nullptr) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    /* the call's last kernel also hands the totals and the error word to pinned (mapped) host
     * memory: both are final here (stream order), and the call needs no copies after it */
    if (id == 0 && tot_h) { *tot_h = *tot_d; *err_h = *err_d; }
    if (id >= n) return;
    const int k = inv[id];
    if (F64) {
        fx[id] = from_fixed(F64[k]); fy[id] = from_fixed(F64[n + k]); fz[id] = from_fixed(F64[2 * n + k]);
    } else {
        fx[id] = F32[k] + F32[3 * (size_t)n + k];
        fy[id] = F32[n + k] + F32[4 * (size_t)n + k];
        fz[id] = F32[2 * n + k] + F32[5 * (size_t)n + k];
    }
    if (cnt_u) cnt_u[id] = cnt_s[k];
}

/* The raw int64 accumulators in user order (x, y, z planes of n), for partial evaluations that
 * are summed exactly (spatial decomposition). */
static __global__ void k_unsort_fixed(int n, const int *__restrict__ inv, const unsigned long long *__restrict__ F64,
                                      long long *__restrict__ out) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    const int k = inv[id];
    out[id] = (long long)F64[k];
    out[(size_t)n + id] = (long long)F64[(size_t)n + k];
    out[2 * (size_t)n + id] = (long long)F64[2 * (size_t)n + k];
}

/* ------------------------------------------------------------------------------------------ */
/* Motion update on cell-sorted state.                                                         */

__device__ __forceinline__ float wrap_pos(float x, float L) {
    if (x < 0.0f) x = __fadd_rn(x, L);
    else if (x >= L) x = __fsub_rn(x, L);
    if (!(x >= 0.0f && x < L)) {
        x = __fsub_rn(x, __fmul_rn(L, floorf(__fdiv_rn(x, L))));
        if (!(x >= 0.0f && x < L)) x = 0.0f;
    }
    return x;
}

__device__ __forceinline__ float force_of(const unsigned long long *F64, const float *F32, int n,
                                          int k, int d) {
    /* FP32 accumulation keeps a high and a low (compensation) plane; the low one is zero in
     * the plain FP32-atomic mode */
    return F64 ? from_fixed(F64[(size_t)d * n + k]) : F32[(size_t)d * n + k] + F32[(size_t)(d + 3) * n + k];
}

/* v += F * cm[type] (half or full kick), x += v * dt, wrap, and bin the new position. */
static __global__ void k_kick_drift_bin(int n, float4 *__restrict__ pos, float4 *__restrict__ vel,
                                 const int *__restrict__ ptype,
                                 const unsigned long long *__restrict__ F64,
                                 const float *__restrict__ F32, const MassTab *__restrict__ mt, float dt, Geom g,
                                 int *__restrict__ cell_of, int *__restrict__ slot,
                                 int *__restrict__ count, unsigned *__restrict__ key) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float cm = mt->cm[ptype[k]];
    float4 v = vel[k];
    float4 p = pos[k];
    v.x = __fmaf_rn(force_of(F64, F32, n, k, 0), cm, v.x);
    v.y = __fmaf_rn(force_of(F64, F32, n, k, 1), cm, v.y);
    v.z = __fmaf_rn(force_of(F64, F32, n, k, 2), cm, v.z);
    p.x = wrap_pos(__fmaf_rn(v.x, dt, p.x), g.L[0]);
    p.y = wrap_pos(__fmaf_rn(v.y, dt, p.y), g.L[1]);
    p.z = wrap_pos(__fmaf_rn(v.z, dt, p.z), g.L[2]);
    vel[k] = v;
    pos[k] = p;
    const int c = cell_of_pos(g, p.x, p.y, p.z);
    cell_of[k] = c;
    key[k] = cell_morton(g, p.x, p.y, p.z, c);
    slot[k] = cell_slot(count, c);
}

/* Reorder the state into the new cell order and clear the force accumulators. */
static __global__ void k_gather_state(int n, const int *__restrict__ sorted,
                               const float4 *__restrict__ pos0, const float4 *__restrict__ vel0,
                               const int *__restrict__ type0, const int *__restrict__ id0,
                               float4 *__restrict__ pos1, float4 *__restrict__ vel1,
                               int *__restrict__ type1, int *__restrict__ id1,
                               unsigned long long *__restrict__ F64, float *__restrict__ F32,
                               int *__restrict__ counts = nullptr) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (counts) counts[k] = 0;
    const int o = sorted[k];
    pos1[k] = pos0[o];
    vel1[k] = vel0[o];
    type1[k] = type0[o];
    id1[k] = id0[o];
    if (F64) { F64[k] = 0ull; F64[n + k] = 0ull; F64[2 * n + k] = 0ull; }
    if (F32) {
#pragma unroll
        for (int d = 0; d < 6; ++d) F32[(size_t)d * n + k] = 0.0f;   /* hi planes 0-2, lo planes 3-5 */
    }
}

/* ---- small systems ----------------------------------------------------------------------------
 * Binning in one launch for systems of at most kSmallN particles and kSmallCells cells: one CTA bins,
 * scans, sorts and gathers, with the counts and keys in shared memory, where the general path takes
 * five launches of ~3.5 us each that do almost nothing (1,728 atoms: 18 -> 8 us per step).  The order
 * is the general path's: by (key, index) inside a cell.  Larger systems need more than one SM. */
constexpr int kSmallN = 4096, kSmallCells = 4096, kSmallThreads = 1024, kSmallPer = kSmallN / kSmallThreads;

struct SmallShared {
    int count[kSmallCells];                  /* occupancy, then the cell's start */
    unsigned long long key[kSmallN];         /* (key, index), cell by cell */
    unsigned short cell[kSmallN];            /* the cell of each entry */
    unsigned short at[kSmallN];              /* cell-order position by index */
    int warp_max[kSmallThreads / 32];
    union { int i[kSmallThreads / 32]; unsigned long long u[kSmallThreads / 32]; } warp_sum;
    unsigned tile_start[kSmallCells];        /* first tiles of the two kinds, 16 bits each */
};

/* Cell-order position of each of the thread's particles (index threadIdx.x + p * kSmallThreads, cell[p],
 * key[p]); fills start[], tot->max_occ and, if wanted, the tiles. */
template <bool TILES>
__device__ __forceinline__ void small_sort(SmallShared &s, int n, int ncells, const int (&cell)[kSmallPer],
                                           const unsigned (&key)[kSmallPer], int (&at)[kSmallPer],
                                           int *__restrict__ start, DevTotals *tot, const Tiles &tl = Tiles()) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int k = t; k < ncells; k += kSmallThreads) s.count[k] = 0;
    __syncthreads();
    int slot[kSmallPer];
#pragma unroll
    for (int p = 0; p < kSmallPer; ++p)
        if (t + p * kSmallThreads < n) slot[p] = atomicAdd(&s.count[cell[p]], 1);
    __syncthreads();
    /* exclusive scan, 4 cells per thread; with tiles, of counts and both kinds of tiles together (at most
     * 4,096 + 256 each, 20 bits) */
    int c[4], mx = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c[k] = 4 * t + k < ncells ? s.count[4 * t + k] : 0;
        mx = max(mx, c[k]);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) s.warp_max[warp] = mx;
    if (TILES) {
        unsigned long long v[4], own = 0ull, carry = 0ull;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = (unsigned)c[k] | ((unsigned long long)cell_tiles(c[k], tl.groups & 0xff) << 20) |
                   ((unsigned long long)cell_tiles(c[k], tl.groups >> 8) << 40);
            own += v[k];
        }
        unsigned long long f = block_scan(own, carry, s.warp_sum.u);
#pragma unroll
        for (int k = 0; k < 4; ++k, f += v[k - 1]) {
            if (4 * t + k >= ncells) continue;
            const int first = (int)(f & 0xfffffu);
            const int2 to = make_int2((int)(f >> 20) & 0xfffff, (int)(f >> 40));
            s.count[4 * t + k] = first;
            start[4 * t + k] = first;
            s.tile_start[4 * t + k] = (unsigned)to.x | ((unsigned)to.y << 16);
            tl.start[4 * t + k] = to;
        }
        if (t == 0) tl.start[ncells] = make_int2((int)(carry >> 20) & 0xfffff, (int)(carry >> 40));
    } else {
        int carry = 0, first = block_scan(c[0] + c[1] + c[2] + c[3], carry, s.warp_sum.i);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (4 * t + k < ncells) { s.count[4 * t + k] = first; start[4 * t + k] = first; }
            first += c[k];
        }
    }
    mx = __reduce_max_sync(0xffffffffu, s.warp_max[lane]);
    if (t == 0) { start[ncells] = n; tot->max_occ = mx; tot->pairs = tot->below = 0ull; }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < kSmallPer; ++p) {
        const int i = t + p * kSmallThreads;
        if (i < n) {
            const int e = s.count[cell[p]] + slot[p];
            s.key[e] = ((unsigned long long)key[p] << 32) | (unsigned)i;
            s.cell[e] = (unsigned short)cell[p];
        }
    }
    __syncthreads();
    /* rank of an entry = the smaller ones of its cell.  By entry, not by particle: neighbouring lanes
     * then walk the same cell, and a load serves them all (by particle, 64 per cell: 52 us) */
#pragma unroll
    for (int p = 0; p < kSmallPer; ++p) {
        const int e = t + p * kSmallThreads;
        if (e >= n) continue;
        const unsigned long long me = s.key[e];
        const int cl = s.cell[e], a = s.count[cl], b = cl + 1 < ncells ? s.count[cl + 1] : n;
        if (TILES) {      /* entry u of a cell writes tile u (a tile has at least one particle) */
            const unsigned to = s.tile_start[cl];
            if (e - a < cell_tiles(b - a, tl.groups & 0xff)) tl.tile[0][(to & 0xffffu) + e - a] = make_int2(cl, e - a);
            if (e - a < cell_tiles(b - a, tl.groups >> 8)) tl.tile[1][(to >> 16) + e - a] = make_int2(cl, e - a);
        }
        int rank = 0;
#pragma unroll 4
        for (int q = a; q < b; ++q) rank += s.key[q] < me;
        s.at[(unsigned)me] = (unsigned short)(a + rank);
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < kSmallPer; ++p)
        if (t + p * kSmallThreads < n) at[p] = s.at[t + p * kSmallThreads];
}

__device__ __forceinline__ void clear_force(int n, int k, unsigned long long *F64, float *F32, int *counts) {
    if (F64) { F64[k] = 0ull; F64[n + k] = 0ull; F64[2 * n + k] = 0ull; }
    if (F32) {
#pragma unroll
        for (int d = 0; d < 6; ++d) F32[(size_t)d * n + k] = 0.0f;   /* hi planes 0-2, lo planes 3-5 */
    }
    if (counts) counts[k] = 0;
}

/* User-order inputs (device memory, or host memory the device reads) into cell order: k_bin_user, k_scan,
 * k_scatter, k_cell_sort and k_gather_user in one, in the list kernel's order and with its tiles or in the
 * other kernels' order.  Also clears the error word and the item counters. */
template <bool LIST>
static __global__ void __launch_bounds__(kSmallThreads)
k_small_user(int n, const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
             const float *__restrict__ q, const int *__restrict__ type, Geom g, int ncells,
             float4 *__restrict__ pos, int *__restrict__ ptype, int *__restrict__ pid, int *__restrict__ inv,
             unsigned long long *__restrict__ F64, float *__restrict__ F32, int *__restrict__ counts, int ntypes,
             int *__restrict__ start, DevTotals *tot, int *__restrict__ work, unsigned *__restrict__ err, Tiles tl) {
    extern __shared__ float4 small_sm[];
    SmallShared &s = *reinterpret_cast<SmallShared *>(small_sm);
    __shared__ unsigned s_err;
    if (threadIdx.x == 0) s_err = 0u;
    if (threadIdx.x < 2) work[threadIdx.x] = 0;
    __syncthreads();
    float4 p[kSmallPer];
    int ty[kSmallPer], cell[kSmallPer], at[kSmallPer];
    unsigned key[kSmallPer];
#pragma unroll
    for (int k = 0; k < kSmallPer; ++k) {
        const int i = threadIdx.x + k * kSmallThreads;
        if (i >= n) continue;
        p[k] = make_float4(x[i], y[i], z[i], q ? q[i] : 0.0f);
        ty[k] = type ? type[i] : 0;
    }
#pragma unroll
    for (int k = 0; k < kSmallPer; ++k) {
        const int i = threadIdx.x + k * kSmallThreads;
        if (i >= n) continue;
        if (!in_box(g, p[k].x, p[k].y, p[k].z)) atomicOr(&s_err, kErrPosition);
        if (ty[k] < 0 || ty[k] >= ntypes) { atomicOr(&s_err, kErrType); ty[k] = 0; }
        cell[k] = cell_of_pos(g, p[k].x, p[k].y, p[k].z);
        key[k] = LIST ? cell_hilbert(g, p[k].x, p[k].y, p[k].z, cell[k]) : cell_morton(g, p[k].x, p[k].y, p[k].z, cell[k]);
    }
    small_sort<LIST>(s, n, ncells, cell, key, at, start, tot, tl);
#pragma unroll
    for (int k = 0; k < kSmallPer; ++k) {
        const int i = threadIdx.x + k * kSmallThreads;
        if (i >= n) continue;
        pos[at[k]] = p[k];
        ptype[at[k]] = ty[k];
        pid[at[k]] = i;
        if (inv) inv[i] = at[k];
        clear_force(n, i, F64, F32, counts);
    }
    if (threadIdx.x == 0) *err = s_err;
}

/* One step's first kick, drift and re-binning of the state: k_kick_drift_bin, k_scan, k_scatter,
 * k_cell_sort and k_gather_state in one. */
static __global__ void __launch_bounds__(kSmallThreads)
k_small_state(int n, const float4 *__restrict__ pos0, const float4 *__restrict__ vel0, const int *__restrict__ type0,
              const int *__restrict__ id0, const MassTab *__restrict__ mt, float dt, Geom g, int ncells,
              float4 *__restrict__ pos1, float4 *__restrict__ vel1, int *__restrict__ type1, int *__restrict__ id1,
              unsigned long long *F64, float *F32, int *__restrict__ counts, int *__restrict__ start, DevTotals *tot,
              int *__restrict__ work) {
    extern __shared__ float4 small_sm[];
    SmallShared &s = *reinterpret_cast<SmallShared *>(small_sm);
    if (threadIdx.x < 2) work[threadIdx.x] = 0;
    float4 p[kSmallPer], v[kSmallPer];
    int ty[kSmallPer], id[kSmallPer], cell[kSmallPer], at[kSmallPer];
    unsigned key[kSmallPer];
#pragma unroll
    for (int q = 0; q < kSmallPer; ++q) {
        const int k = threadIdx.x + q * kSmallThreads;
        if (k >= n) continue;
        ty[q] = type0[k];
        id[q] = id0[k];
        v[q] = vel0[k];
        p[q] = pos0[k];
        const float cm = mt->cm[ty[q]];
        v[q].x = __fmaf_rn(force_of(F64, F32, n, k, 0), cm, v[q].x);
        v[q].y = __fmaf_rn(force_of(F64, F32, n, k, 1), cm, v[q].y);
        v[q].z = __fmaf_rn(force_of(F64, F32, n, k, 2), cm, v[q].z);
        p[q].x = wrap_pos(__fmaf_rn(v[q].x, dt, p[q].x), g.L[0]);
        p[q].y = wrap_pos(__fmaf_rn(v[q].y, dt, p[q].y), g.L[1]);
        p[q].z = wrap_pos(__fmaf_rn(v[q].z, dt, p[q].z), g.L[2]);
        cell[q] = cell_of_pos(g, p[q].x, p[q].y, p[q].z);
        key[q] = cell_morton(g, p[q].x, p[q].y, p[q].z, cell[q]);
        clear_force(n, k, F64, F32, counts);     /* the thread's own entries, read above */
    }
    small_sort<false>(s, n, ncells, cell, key, at, start, tot);
#pragma unroll
    for (int q = 0; q < kSmallPer; ++q) {
        if ((int)threadIdx.x + q * kSmallThreads >= n) continue;
        pos1[at[q]] = p[q];
        vel1[at[q]] = v[q];
        type1[at[q]] = ty[q];
        id1[at[q]] = id[q];
    }
}

/* Second half kick (velocity Verlet) and, when asked, per-block kinetic-energy partials
 * (FP32 per particle and within the block, in a fixed order; FP64 across blocks). */
static __global__ void __launch_bounds__(256) k_kick(int n, float4 *__restrict__ vel, const int *__restrict__ ptype,
                                                     const unsigned long long *__restrict__ F64,
                                                     const float *__restrict__ F32, const MassTab *__restrict__ mt, int do_kick,
                                                     double *__restrict__ kepart) {
    __shared__ float s_k[8];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    float ke = 0.0f;
    if (k < n) {
        const int t = ptype[k];
        float4 v = vel[k];
        if (do_kick) {
            const float cm = mt->cm[t];
            v.x = __fmaf_rn(force_of(F64, F32, n, k, 0), cm, v.x);
            v.y = __fmaf_rn(force_of(F64, F32, n, k, 1), cm, v.y);
            v.z = __fmaf_rn(force_of(F64, F32, n, k, 2), cm, v.z);
            vel[k] = v;
        }
        /* 1/2 m v^2 in kcal/mol with v in A/fs and m in amu: divide by 4.184e-4. */
        if (kepart) ke = 0.5f * mt->mass[t] * (v.x * v.x + v.y * v.y + v.z * v.z) * (1.0f / 4.184e-4f);
    }
    if (!kepart) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ke += __shfl_xor_sync(0xffffffffu, ke, o);
    if ((threadIdx.x & 31) == 0) s_k[threadIdx.x >> 5] = ke;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b += s_k[w];
        kepart[blockIdx.x] = b;
    }
}

/* Sorted state back to user order. */
static __global__ void k_unsort_state(int n, const int *__restrict__ pid, const float4 *__restrict__ pos,
                               const float4 *__restrict__ vel, float *__restrict__ x,
                               float *__restrict__ y, float *__restrict__ z, float *__restrict__ vx,
                               float *__restrict__ vy, float *__restrict__ vz) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int id = pid[k];
    const float4 p = pos[k], v = vel[k];
    x[id] = p.x; y[id] = p.y; z[id] = p.z;
    vx[id] = v.x; vy[id] = v.y; vz[id] = v.z;
}

/* Gather user-order velocities into cell order (set_state). */
static __global__ void k_gather_vel(int n, const int *__restrict__ pid, const float *__restrict__ vx,
                             const float *__restrict__ vy, const float *__restrict__ vz,
                             float4 *__restrict__ vel) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int id = pid[k];
    vel[k] = vx ? make_float4(vx[id], vy[id], vz[id], 0.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
}

/* ------------------------------------------------------------------------------------------ */
/* Per-pair evaluation: the drop-in for the OpenCL library function RL_LJ_Evaluation.          */

template <int ORDER, bool SEP>
static __global__ void k_pair_eval(int n, const float4 *__restrict__ ref, const float4 *__restrict__ nbr,
                            const int *__restrict__ tref, const int *__restrict__ tnbr, Geom g,
                            TableDev tab, const float4 *__restrict__ pcoef, int ntypes, float ke,
                            float4 *__restrict__ out, float2 *__restrict__ aux, int exact) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 a = ref[k], b = nbr[k];
    const int ta = tref ? tref[k] : 0, tb = tnbr ? tnbr[k] : 0;
    float dx, dy, dz;
    if (exact) {
        dx = wrap_exact(a.x, b.x, g.L[0], g.h[0]);
        dy = wrap_exact(a.y, b.y, g.L[1], g.h[1]);
        dz = wrap_exact(a.z, b.z, g.L[2], g.h[2]);
    } else {
        dx = wrap_d(__fsub_rn(a.x, b.x), g.L[0], g.h[0]);
        dy = wrap_d(__fsub_rn(a.y, b.y), g.L[1], g.h[1]);
        dz = wrap_d(__fsub_rn(a.z, b.z), g.L[2], g.h[2]);
    }
    const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    float fs = 0.0f;
    if (r2 > 0.0f && r2 <= g.rc2) {
        const bool coul = ke != 0.0f;
        float v14, v8, v3, v12, v6, v1;
        int below;
        pair_functions<ORDER, SEP, false>(tab, r2, coul, v14, v8, v3, v12, v6, v1, below);
        const float4 pc = pcoef[ta * ntypes + tb];
        const float qq = __fmul_rn(__fmul_rn(ke, a.w), b.w);
        fs = combine_force<SEP>(pc, qq, coul, v14, v8, v3);
        o = make_float4(__fmul_rn(fs, dx), __fmul_rn(fs, dy), __fmul_rn(fs, dz), 0.0f);
    }
    out[k] = o;
    if (aux) aux[k] = make_float2(r2, fs);
}

}  // namespace mdrl
