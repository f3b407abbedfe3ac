/*
 * mdrl_force_list.cuh — the half-shell pair-force kernel of force evaluations, over particle lists
 * (sm_103a).
 *
 * Work item = (tile of a home cell, column class).  The 14 half-shell cells of a home cell
 * (SC/Particle_Pair_Gen_HalfShell.v:14-24) are 5 columns of cells along z -- (0,0): the home cell and
 * the one above; (0,1), (1,-1), (1,0), (1,1): three cells each -- and cells that follow one another in
 * z follow one another in the cell-sorted arrays, so a column is one contiguous range of particles
 * plus, at the z faces of the box, one wrapped cell.  Classes: (0,0); (1,0) with its two diagonal
 * neighbours; (0,1).  The home cell's particles are cut into groups of 4 (consecutive on the in-cell
 * Hilbert curve, so compact in space) and these into even tiles of at most 4 or 8 groups, which the binning
 * numbers and writes down (Tiles in mdrl_kernels.cuh): a launch has as many items as there are tiles,
 * however unevenly the cells are filled.  (Items by the mean occupancy: a droplet of 13,000 atoms in a
 * 200 A box 1,250 us, 60,000 in 300 A 19.95 ms; now 207 us and 0.95 ms, evenly filled systems alike.)
 * Per item one warp
 *   1. lists the class's particles that lie within rc of the tile's bounding box (one lane per
 *      particle, ballot + popc compaction);
 *   2. marks, per listed particle, the groups whose bounding box it is within rc of: 2 in 3 of the
 *      (i, j) candidates that remain are pairs (92k system; of the 4 x 8 blocks that the per-item
 *      kernel of mdrl_force_warp.cuh culls, 1 in 3 are);
 *   3. per group, takes 32 marked particles at a time, one per lane, against the group's 4
 *      i-particles, which are the same in every lane.  Only the table loads depend on the filter
 *      0 < r2 <= rc2; a rejected candidate's scalar force is selected to 0.  The j force of the 4 is
 *      added to the warp's accumulator in shared memory (a lane owns its j: no shuffles), and the i
 *      forces stay in registers until the group's list ends (one reduce-scatter, then to the global
 *      accumulators: kept in shared memory until a run of lists ends they would be FP32 sums over
 *      any number of cells);
 *   4. adds the list's j forces to the global accumulators (one atomic per particle and component).
 *      So no FP32 sum holds more than one list's 256 j, or one tile's 32 i.
 * The two levels of lists only drop candidates that cannot be pairs: the box test of
 * mdrl_force_warp.cuh (tests/test_cull_bound.py) with one particle for the second box.  So the accepted
 * pairs are those of the plain traversal, bit for bit.  Deterministic: every FP32 partial sum is of one
 * tile and one list, whose order follows from the particles of its cells alone, and the int64
 * global sums are exact; so the result does not depend on scheduling or on what else a launch
 * holds (other replicas, other slabs), nor on whether the items are fine (below).
 *
 * The grid is persistent: as many CTAs as fit, 4 independent warps each, which share the type-pair
 * multipliers; a warp takes the next item from a counter.  The class whose items are shortest runs
 * last.  A launch with few items runs fine ones: an item is one run, and the 4 warps of a CTA share it,
 * one group each.
 *
 * What bounds it (92k system, order 2, exact rule: 283 us, 362 us for the kernel it replaces; 1M system
 * 1.74 ms, 2.61; order 1 92k 260 us): the L1 data pipe, 73 % busy at 92k and 82 % at 1M
 * under the profiler, most of it on the table gathers.  An earlier build timed
 * without parts: no table 210 us (at 299), no c2 gather of r^-3 274, no j accumulation 278, no i
 * reduction 284, no atomics 290, lists alone 77.  The gathers of one table element are therefore
 * kept in arrays of their own: 16-byte elements at a 32-byte stride use half the banks (299 -> 276 us
 * with the 13-shuffle reduction and the prefetch of the next block's positions).  20 warps per SM at 96
 * registers: 16 at 128 are 2-5 % slower.  What a phase does not need is kept in shared memory, or the
 * pair loop spills.
 */
#pragma once

#include <algorithm>

#include "mdrl_force_warp.cuh"

namespace mdrl {

constexpr int kWarpsPerCta = 4;               /* independent warps of a CTA */
constexpr int kListCtas = 5;                  /* resident CTAs the registers (96) allow */
constexpr int kListCap = 256;                 /* tile-list entries (a byte indexes them) */
constexpr int kListBlocks = kListCap / 32;    /* its blocks of 32: one mask byte each in two registers */
static_assert(kListCap % 32 == 0 && kListBlocks <= 8, "");
constexpr int kTileGroups = 8;                /* most groups of 4 i-particles in a tile */
constexpr int kClasses = 3;                   /* column classes of the half shell */
constexpr int kMaxCols = 3;                   /* columns of a class */

/* The classes' columns, by the first half-shell offset of each: (0,0); (1,0), (1,-1), (1,1); (0,1).
 * The two diagonal columns hold few particles within reach, so they share the lists of the column
 * between them. */
__constant__ int c_class_cols[kClasses] = {1, 3, 1};
__constant__ int c_class_first[kClasses][kMaxCols] = {{0, 0, 0}, {8, 5, 11}, {2, 2, 2}};

/* Runs of a column class: its ranges that share a periodic shift, and so a list (at most 3 columns
 * by 2).  FINE items are one run each; the (class, run) of each in launch order. */
constexpr int kRuns = 6, kFineRuns = 10;
__constant__ int c_fine_class[kFineRuns] = {0, 1, 2, 0, 1, 1, 1, 1, 1, 2};
__constant__ int c_fine_run[kFineRuns] = {0, 0, 0, 1, 1, 2, 3, 4, 5, 1};

/* Groups per tile of classes 0 and 1 (low byte) and of class 2, whose items run last. */
inline int tile_groups(int ncells) { return ncells < 400 ? 0x404 : (ncells < 2000 ? 0x408 : 0x808); }

constexpr int kFineItems = 16;    /* per SM: below this many whole items a launch runs fine ones */

/* Whether a launch runs FINE items: the 4 warps of a CTA share each (one group of its tile each,
 * tiles of at most 4 groups), and an item is one run. */
inline bool fine_items(int tg, long long items, int num_sms) {
    return (tg & 0xff) <= kWarpsPerCta && (tg >> 8) <= kWarpsPerCta && items <= kFineItems * num_sms;
}

/* Items of a launch over `cells` of a system's ncells cells if its n particles fill them evenly, about one
 * tile each with 10 % to spare: what the choice of FINE items goes by. */
inline long long items_expected(long long n, int ncells, int cells) {
    const int tg = tile_groups(ncells);
    const double groups = 1.1 * 0.25 * (double)n / (ncells > 0 ? ncells : 1);
    return (long long)cells * (2 * ((int)(groups / (tg & 0xff)) + 1) + (int)(groups / (tg >> 8)) + 1);
}

/* The most tiles of tg groups that n particles in ncells cells can make, and the most items of a launch
 * over them: its result slots. */
inline long long tiles_max(long long n, int ncells, int tg) { return n / (4 * tg) + (n < ncells ? n : ncells); }
inline long long items_max(long long n, int ncells, bool fine) {
    const int tg = tile_groups(ncells);
    const long long t0 = tiles_max(n, ncells, tg & 0xff);
    return fine ? kFineRuns * t0 : 2 * t0 + tiles_max(n, ncells, tg >> 8);
}

/* Gathers of one table element per lane, issued only by the lanes whose candidate the filter accepted
 * (p): the L1 data pipe, which these gathers load most, spends wavefronts on active lanes (92k
 * launch, order 2: 338 us with every lane loading a clamped row, 323 us so).  The zero is what keeps
 * the load in a block of its own: with it left out the compiler predicates the loads of all 4
 * candidates at once, and the registers they need spill (630 us). */
template <class V>
__device__ __forceinline__ V ldg_if(const V *a, bool p) {
    V v = {};
    if (p) v = __ldg(a);
    return v;
}

/* The pair functions at r2e (clamped into the table) for the lanes with p; the arithmetic of
 * pair_functions_fast.  Order 1 reads a 16- and an 8-byte element, order 2 the packed 36-byte rows
 * (a smaller L1 footprint than 48), order 3 float4 rows. */
template <int ORDER, bool SEP, bool ENERGY, bool COUL>
__device__ __forceinline__ void pair_functions_if(const TableDev &t, float r2e, bool p, float &v14, float &v8,
                                                  float &v3, float &v12, float &v6, float &v1) {
    if (ORDER == 0) {
        int below;
        pair_functions<0, SEP, ENERGY>(t, r2e, COUL, v14, v8, v3, v12, v6, v1, below);
        return;
    }
    const unsigned bits = __float_as_uint(r2e);
    const int idx = (int)(bits >> (23 - t.lb)) - ((127 + t.min_log2) << t.lb);
    if (ORDER == 1) {
        const float4 a = ldg_if(t.wa + idx, p);
        v14 = madd<SEP>(a.y, r2e, a.x);
        v8 = madd<SEP>(a.w, r2e, a.z);
        if (COUL) { const float2 c = ldg_if(t.wc + idx, p); v3 = madd<SEP>(c.y, r2e, c.x); }
        if (ENERGY) {
            const float2 d = ldg_if(t.e2 + 3 * idx, p), e = ldg_if(t.e2 + 3 * idx + 1, p);
            v12 = madd<SEP>(d.y, r2e, d.x);
            v6 = madd<SEP>(e.y, r2e, e.x);
            if (COUL) { const float2 f = ldg_if(t.e2 + 3 * idx + 2, p); v1 = madd<SEP>(f.y, r2e, f.x); }
        }
        return;
    }
    /* table_variable without its branch: the mask is 0 in the monomial form */
    const float x = __fsub_rn(r2e, __uint_as_float(bits & t.bmask));
    if (ORDER == 2) {
        const float4 a = ldg_if(t.wa + idx, p), b = ldg_if(t.wb + idx, p);
        v14 = madd<SEP>(madd<SEP>(a.z, x, a.y), x, a.x);
        v8 = madd<SEP>(madd<SEP>(b.y, x, b.x), x, a.w);
        if (COUL) v3 = madd<SEP>(madd<SEP>(ldg_if(t.w1 + idx, p), x, b.w), x, b.z);
    } else {
        v14 = poly4<ORDER, SEP>(ldg_if(t.f4 + 3 * idx, p), x);
        v8 = poly4<ORDER, SEP>(ldg_if(t.f4 + 3 * idx + 1, p), x);
        if (COUL) v3 = poly4<ORDER, SEP>(ldg_if(t.f4 + 3 * idx + 2, p), x);
    }
    if (ENERGY) {
        v12 = poly4<ORDER, SEP>(ldg_if(t.e4 + 3 * idx, p), x);
        v6 = poly4<ORDER, SEP>(ldg_if(t.e4 + 3 * idx + 1, p), x);
        if (COUL) v1 = poly4<ORDER, SEP>(ldg_if(t.e4 + 3 * idx + 2, p), x);
    }
}

/* One warp's shared memory. */
template <bool EXTRA>
struct ListSmem {
    float4 i[32];                        /* tile: x, y, z (shifted), ke q */
    float4 g[kTileGroups][2];            /* group boxes: centre, half widths + margin (far: empty) */
    float fj[3][kListCap];               /* j accumulator of the tile list */
    int it[32];                          /* tile: type * ntypes */
    int idx[kListCap];                   /* tile list: particle */
    unsigned char list[kListCap];        /* the current group's list: tile-list entries */
    /* the item's, tile's and column range's state: read back from here between the phases, so that
     * the pair loop has the registers */
    int hs, ni, hx, hy, hz, cls, i0, i1, ngr;
    int cbase[kMaxCols];                 /* first cell of each column */
    float sx, sy[kMaxCols];              /* the columns' x and y shifts */
    int range, jb, je, self, total, run, want;
    float csy, csz;                      /* the current range's y and z shifts */
    float tc[3], th[3];                  /* tile box: centre, half widths + margin */
    float js[3];                         /* exact rule: taken off the j coordinates */
    float sd[3];                         /* kDiffShift: added to every difference */
    int next;                            /* the CTA's item when its warps share items */
    unsigned pairs, below;               /* sums of a warp that shares its items */
    int ci[EXTRA ? 32 : 1];              /* partner counts (energy launches) */
    int cj[EXTRA ? kListCap : 1];
    double e[EXTRA ? 3 : 1];             /* energies and virial of a warp that shares its items */
};

inline size_t force_list_smem_bytes(int ntypes, bool extra) {
    const size_t t2 = (size_t)((ntypes * ntypes + 1) & ~1);
    return sizeof(float2) * t2 * (extra ? 2 : 1) +
           kWarpsPerCta * (extra ? sizeof(ListSmem<true>) : sizeof(ListSmem<false>));
}

/* The tiles of a launch: of kind 0 tile[0][first->x .. last->x), of kind 1 tile[1][first->y .. last->y);
 * groups per tile as Tiles::groups (a batch: its replicas').  Items, in launch order: the tiles of kind 0
 * for class 0, for class 1, those of kind 1 for class 2; FINE (one kind) one per tile for every run of a
 * class; MODE kDiffWrap one per tile. */
struct ListTiles {
    const int2 *first = nullptr, *last = nullptr;
    const int2 *tile[2] = {nullptr, nullptr};
    int groups = 0;
    const int *rep_of_cell = nullptr;
};

/* The launch signature.  work: the item counter, zero at launch; nitems: receives the number of items. */
typedef void (*list_fn)(const float4 *, const int *, const int *, Geom, TableDev, const float4 *, int, float, int,
                        unsigned long long *, int *, UnitOut *, ListTiles, const BatchRep *, unsigned *, int *, int *,
                        DevTotals *);

/* Cells along an axis that can hold a partner of a particle of cell 0, on either side: 1 as the cells are
 * at least rc wide, 2 where one that is barely so could lose a pair to rounding. */
__device__ __forceinline__ int axis_reach(const Geom &g, int d) { return g.edge[d] * g.edge[d] > 1.00001f * g.rc2 ? 1 : 2; }

/* The cells that the particles of cell (hx, hy, hz) of a replica with minimum images pair with, among the
 * later ones of its storage order: range r of ranges(), cells [z0, z1] of column (cx, cy); false:
 * none.  Two ranges per column of the window around the home cell, the second one for what lies across
 * the z face; the home column starts at the home cell. */
struct WrapWindow {
    int rx, ry, rz, nx, ny;              /* reach; columns of the window along x and y */
    __device__ __forceinline__ WrapWindow(const Geom &g) {
        rx = axis_reach(g, 0); ry = axis_reach(g, 1); rz = axis_reach(g, 2);
        nx = min(g.nc[0], 2 * rx + 1);
        ny = min(g.nc[1], 2 * ry + 1);
    }
    __device__ __forceinline__ int ranges() const { return 2 * nx * ny; }
    __device__ __forceinline__ bool range(const Geom &g, int hx, int hy, int hz, int r, int &col, int &z0, int &z1) const {
        const int k = r >> 1, ix = k / ny, iy = k - ix * ny;
        int cx = ix, cy = iy;
        if (nx < g.nc[0]) { cx = hx - rx + ix; cx += cx < 0 ? g.nc[0] : (cx >= g.nc[0] ? -g.nc[0] : 0); }
        if (ny < g.nc[1]) { cy = hy - ry + iy; cy += cy < 0 ? g.nc[1] : (cy >= g.nc[1] ? -g.nc[1] : 0); }
        const int home = hx * g.nc[1] + hy, nz = g.nc[2];
        col = cx * g.nc[1] + cy;
        if (col < home) return false;
        const int lo = hz - rz, hi = hz + rz;
        const bool whole = nz <= 2 * rz + 1;
        if (!(r & 1)) {
            z0 = col == home ? hz : (whole ? 0 : max(lo, 0));
            z1 = whole ? nz - 1 : min(hi, nz - 1);
            return true;
        }
        if (whole) return false;
        if (lo < 0) { z0 = nz + lo; z1 = nz - 1; return true; }       /* later than the home cell in any column */
        z0 = 0; z1 = hi - nz;
        return hi >= nz && col != home;
    }
};

/* Warp-wide minimum and maximum of floats. */
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

/* Sum over the 32 lanes of v[0..11], scattered: on return lane 8 k + 2 c (and its odd neighbour)
 * holds in v[0] the sum of the input v[3 k + c], c < 3 (13 shuffles). */
__device__ __forceinline__ void reduce_scatter12(float (&v)[12], int lane) {
    const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4, b2 = lane & 2;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
        const float send = b16 ? v[t] : v[6 + t];
        const float keep = b16 ? v[6 + t] : v[t];
        v[t] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const float send = b8 ? v[t] : v[3 + t];
        const float keep = b8 ? v[3 + t] : v[t];
        v[t] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    {   /* components 0, 1 to the lower four lanes of an octet, component 2 to the upper four */
        const float s0 = b4 ? v[0] : v[2], s1 = v[1];
        const float r0 = __shfl_xor_sync(0xffffffffu, s0, 4), r1 = __shfl_xor_sync(0xffffffffu, s1, 4);
        v[0] = (b4 ? v[2] : v[0]) + r0;
        v[1] = s1 + r1;
    }
    {   /* component 1 to lanes 2, 3; lanes 6, 7 repeat component 2 */
        const float send = b2 ? v[0] : (b4 ? v[0] : v[1]);
        const float keep = b4 ? v[0] : (b2 ? v[1] : v[0]);
        v[0] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
}

/* hi + lo in FP64; an infinite or NaN hi by itself, whose lo is NaN. */
__device__ __forceinline__ double hi_lo(float hi, float lo) { return isfinite(hi) ? (double)hi + lo : (double)hi; }

/* BATCH: the tiles are those of a batch's replicas (replica geometry, cell offset and tile groups from
 * reps); with MODE kDiffWrap of replicas whose edges all exceed 2 rc: a tile's particles against the later
 * ones of the cells within reach (WrapWindow). */
template <int ORDER, bool SEP, bool EXTRA, int MODE, bool COUL, bool FINE, bool BATCH = false>
__global__ void __launch_bounds__(32 * kWarpsPerCta, EXTRA ? 4 : kListCtas)
k_force_list(const float4 *__restrict__ pos, const int *__restrict__ ptype, const int *__restrict__ cstart,
             Geom gparam, TableDev tab, const float4 *__restrict__ pcoef, int ntypes, float ke, int n,
             unsigned long long *__restrict__ F64, int *__restrict__ counts, UnitOut *__restrict__ uout,
             ListTiles lt, const BatchRep *__restrict__ reps, unsigned *__restrict__ err, int *__restrict__ work,
             int *__restrict__ nitems_out, DevTotals *tot) {
    constexpr bool kCellPair = BATCH && MODE == kDiffWrap;
    const int2 tile0 = *lt.first, tile1 = *lt.last;
    const int t2 = (ntypes * ntypes + 1) & ~1;
    extern __shared__ float4 wsm[];
    float2 *sCoefF = reinterpret_cast<float2 *>(wsm);           /* (A14, B8) [T^2] */
    float2 *sCoefE = sCoefF + t2;                               /* (A12, B6) [T^2], EXTRA only */
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ListSmem<EXTRA> *const all = reinterpret_cast<ListSmem<EXTRA> *>(sCoefE + (EXTRA ? t2 : 0));
    ListSmem<EXTRA> &s = all[warp];
    for (int t = threadIdx.x; t < ntypes * ntypes; t += 32 * kWarpsPerCta) {
        const float4 c4 = pcoef[t];
        sCoefF[t] = make_float2(c4.x, c4.y);
        if (EXTRA) sCoefE[t] = make_float2(c4.z, c4.w);
    }
    __syncthreads();

    const int nt = tile1.x - tile0.x;
    const int nitems = kCellPair ? nt : (FINE ? kFineRuns * nt : 2 * nt + (tile1.y - tile0.y));
    if (blockIdx.x == 0 && threadIdx.x == 0) *nitems_out = nitems;

    const float far = 1.0e18f;
    const unsigned below = (1u << lane) - 1u;

    unsigned long long pairs_sum = 0;    /* lane 0: the warp's items' */
    /* the next item of this warp; FINE: of this CTA, whose first one is that of its own number (the launch is
     * short: the counter's latency would show) */
    auto next = [&]() {
        int b = 0;
        if (FINE) {
            __syncthreads();
            if (threadIdx.x == 0) all[0].next = gridDim.x + atomicAdd(work, 1);
            __syncthreads();
            return all[0].next;
        }
        if (lane == 0) b = atomicAdd(work, 1);
        return __shfl_sync(0xffffffffu, b, 0);
    };
    for (int b = FINE ? blockIdx.x : next(); b < nitems; b = next()) {
        /* item -> class, run, home cell, tile */
        BatchRep rep;
        const Geom &g = BATCH ? rep.g : gparam;
        int coff = 0, tile, ntile;
        {
            int cls = 0, want = -1, tgw = lt.groups;      /* want: the one run of the item, -1: all */
            int2 e;
            if (kCellPair) {
                e = lt.tile[0][tile0.x + b];
                want = FINE ? 0 : -1;
            } else if (FINE) {
                const int q = b / nt;
                cls = c_fine_class[q];
                want = c_fine_run[q];
                e = lt.tile[0][tile0.x + b - q * nt];
            } else {
                cls = b < nt ? 0 : (b < 2 * nt ? 1 : 2);
                e = cls == 2 ? lt.tile[1][tile0.y + b - 2 * nt] : lt.tile[0][tile0.x + b - cls * nt];
            }
            if (BATCH) {
                rep = reps[lt.rep_of_cell[e.x]];
                coff = rep.cell_off;
                tgw = rep.tile_groups;
            }
            const int h = e.x - coff;
            tile = e.y;
            const int hs = cstart[e.x], ni = cstart[e.x + 1] - hs;
            /* the column: cells (cx, cy, hz - 1 .. hz + 1), or the home cell and the one above */
            bool skip = false;
            const int nyz = g.nc[1] * g.nc[2];
            const int hx = h / nyz, hy = (h / g.nc[2]) % g.nc[1], hz = h % g.nc[2];
            if (kCellPair) {
                s.hx = hx;
                s.hy = hy;
            } else {
                int cx = hx + (cls == 1 ? 1 : 0);
                s.sx = cx >= g.nc[0] ? -g.L[0] : 0.0f;
                cx = cx >= g.nc[0] ? cx - g.nc[0] : cx;
                for (int k = 0; k < c_class_cols[cls]; ++k) {
                    int cy = hy + c_halfshell[c_class_first[cls][k]][1];
                    s.sy[k] = cy >= g.nc[1] ? -g.L[1] : (cy < 0 ? g.L[1] : 0.0f);
                    cy = cy < 0 ? cy + g.nc[1] : (cy >= g.nc[1] ? cy - g.nc[1] : cy);
                    const int cbase = coff + (cx * g.nc[1] + cy) * g.nc[2];
                    s.cbase[k] = cbase;
                    /* an overflowing cell (reported by the in-cell sort) skips the item: bounded time */
                    for (int dz = cls ? -1 : 0; dz <= 1; ++dz) {
                        int cz = hz + dz;
                        cz = cz < 0 ? cz + g.nc[2] : (cz >= g.nc[2] ? cz - g.nc[2] : cz);
                        skip = skip || cstart[cbase + cz + 1] - cstart[cbase + cz] > kMaxCellOcc;
                    }
                }
            }
            s.hz = hz;
            s.hs = hs; s.ni = ni; s.cls = cls;
            if (FINE) s.want = want;
            /* the cell's tiles follow from its occupancy alone */
            ntile = skip ? 0 : cell_tiles(ni, cls == 2 ? tgw >> 8 : tgw & 0xff);
        }
        __syncwarp();

        unsigned acc_pairs = 0, acc_below = 0;
        /* energies and virial of the lane over the item: a visit's FP32 sums are added up with their rounding
         * errors beside them (2^-46 of the largest; FP64 runs at 1/64 of the FP32 rate), so that the totals do
         * not depend on how visits are shared among warps and items */
        float ehi[3] = {0.0f, 0.0f, 0.0f}, elo[3] = {0.0f, 0.0f, 0.0f};

        if (ntile) {
            {
                const int ng = (s.ni + 3) >> 2, ga = ng * tile / ntile, gb = ng * (tile + 1) / ntile;
                const int i0 = s.hs + 4 * ga, i1 = min(s.hs + s.ni, s.hs + 4 * gb);
                s.it[lane] = i0 + lane < i1 ? __ldg(ptype + i0 + lane) * ntypes : 0;
                if (EXTRA) s.ci[lane] = 0;
                __syncwarp();
                s.i0 = i0; s.i1 = i1; s.ngr = gb - ga;
                s.range = 0; s.jb = 0; s.je = 0; s.run = -1; s.csy = s.csz = 3.0e38f;
                __syncwarp();
            }
            for (;;) {
                /* ---- 1: the tile list, until it is full, the shift changes or the column ends ---- */
                int cnt = 0;
                {
                    int jb = s.jb, je = s.je;
                    float tcx = s.tc[0], tcy = s.tc[1], tcz = s.tc[2], thx = s.th[0], thy = s.th[1], thz = s.th[2];
                    float jsx = s.js[0], jsy = s.js[1], jsz = s.js[2];
                    float4 pn = make_float4(0.0f, 0.0f, 0.0f, 0.0f);    /* the next block's positions */
                    if (jb + lane < je) pn = __ldg(pos + jb + lane);
                    while (cnt <= kListCap - 32) {
                        if (jb >= je) {
                            /* the next range: the columns' unwrapped cells, then their cells across a z
                             * face */
                            const int range = s.range, ncol = c_class_cols[s.cls];
                            float sy = 0.0f, sz = 0.0f;
                            int lo, hi;
                            bool own = s.cls == 0;
                            if (kCellPair) {
                                const WrapWindow win(g);
                                if (range == win.ranges()) break;
                                int col, z0, z1;
                                lo = hi = 0;
                                own = true;
                                if (win.range(g, s.hx, s.hy, s.hz, range, col, z0, z1)) {
                                    const int c0 = coff + col * g.nc[2];
                                    lo = cstart[c0 + z0];
                                    hi = cstart[c0 + z1 + 1];
                                    for (int z = z0; z <= z1; ++z)     /* an overflowing cell: bounded time */
                                        if (cstart[c0 + z + 1] - cstart[c0 + z] > kMaxCellOcc) hi = lo;
                                }
                            } else if (range == 2 * ncol) {
                                break;
                            } else if (range < ncol) {
                                const int z0 = s.cls ? max(s.hz - 1, 0) : s.hz, z1 = min(s.hz + 1, g.nc[2] - 1);
                                lo = cstart[s.cbase[range] + z0]; hi = cstart[s.cbase[range] + z1 + 1];
                                sy = s.sy[range];
                            } else {
                                own = false;
                                int cz = -1;
                                if (s.hz == g.nc[2] - 1) { cz = 0; sz = -g.L[2]; }
                                else if (s.cls && s.hz == 0) { cz = g.nc[2] - 1; sz = g.L[2]; }
                                lo = cz < 0 ? 0 : cstart[s.cbase[range - ncol] + cz];
                                hi = cz < 0 ? 0 : cstart[s.cbase[range - ncol] + cz + 1];
                                sy = s.sy[range - ncol];
                            }
                            const bool same = s.csy == sy && s.csz == sz;
                            if (lo < hi && cnt > 0 && !same) break;       /* other shift: finish the list first */
                            __syncwarp();
                            s.range = range + 1;
                            __syncwarp();
                            if (lo >= hi) continue;
                            if (FINE && !same) {
                                const int run = s.run + 1;
                                __syncwarp();
                                s.run = run;
                                __syncwarp();
                            }
                            if (FINE && s.run != s.want) {
                                s.csy = sy; s.csz = sz;
                                __syncwarp();
                                continue;
                            }
                            jb = own ? max(lo, s.i0 + 1) : lo;
                            je = hi;
                            if (jb + lane < je) pn = __ldg(pos + jb + lane);
                            if (same) continue;
                            s.self = own;
                            /* the tile under this shift.  Exact rule: the box edge comes off the high
                             * side's coordinates (see pair_diff) */
                            const float sx = kCellPair ? 0.0f : s.sx;
                            const float margin = 9.5367431640625e-07f * fmaxf(g.L[0], fmaxf(g.L[1], g.L[2]));
                            const bool have = s.i0 + lane < s.i1;
                            float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            if (have) p = __ldg(pos + s.i0 + lane);
                            float sdx = 0.0f, sdy = 0.0f, sdz = 0.0f;
                            if (MODE == kDiffExact) {
                                p.x = __fadd_rn(p.x, fminf(sx, 0.0f)); p.y = __fadd_rn(p.y, fminf(sy, 0.0f)); p.z = __fadd_rn(p.z, fminf(sz, 0.0f));
                                jsx = fmaxf(sx, 0.0f); jsy = fmaxf(sy, 0.0f); jsz = fmaxf(sz, 0.0f);
                            }
                            if (MODE == kDiffShift) { sdx = sx; sdy = sy; sdz = sz; }
                            float lx = have ? p.x : 3.0e38f, ly = have ? p.y : 3.0e38f, lz = have ? p.z : 3.0e38f;
                            float ux = have ? p.x : -3.0e38f, uy = have ? p.y : -3.0e38f, uz = have ? p.z : -3.0e38f;
                            s.i[lane] = have ? make_float4(p.x, p.y, p.z, __fmul_rn(ke, p.w)) : make_float4(far, far, far, 0.0f);
#pragma unroll
                            for (int o = 1; o < 4; o <<= 1) {
                                lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o));
                                ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o));
                                lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o));
                                ux = fmaxf(ux, __shfl_xor_sync(0xffffffffu, ux, o));
                                uy = fmaxf(uy, __shfl_xor_sync(0xffffffffu, uy, o));
                                uz = fmaxf(uz, __shfl_xor_sync(0xffffffffu, uz, o));
                            }
                            if ((lane & 3) == 0) {
                                const bool some = lx <= ux;
                                s.g[lane >> 2][0] = make_float4(some ? 0.5f * (lx + ux) + sdx : -far, 0.5f * (ly + uy) + sdy,
                                                                0.5f * (lz + uz) + sdz, 0.0f);
                                s.g[lane >> 2][1] = make_float4(0.5f * (ux - lx) + margin, 0.5f * (uy - ly) + margin,
                                                                0.5f * (uz - lz) + margin, 0.0f);
                            }
                            lx = warp_min(lx); ly = warp_min(ly); lz = warp_min(lz);
                            ux = warp_max(ux); uy = warp_max(uy); uz = warp_max(uz);
                            tcx = 0.5f * (lx + ux) + sdx; tcy = 0.5f * (ly + uy) + sdy; tcz = 0.5f * (lz + uz) + sdz;
                            thx = 0.5f * (ux - lx) + margin; thy = 0.5f * (uy - ly) + margin; thz = 0.5f * (uz - lz) + margin;
                            s.csy = sy; s.csz = sz;
                            s.tc[0] = tcx; s.tc[1] = tcy; s.tc[2] = tcz;
                            s.th[0] = thx; s.th[1] = thy; s.th[2] = thz;
                            s.js[0] = jsx; s.js[1] = jsy; s.js[2] = jsz;
                            s.sd[0] = sdx; s.sd[1] = sdy; s.sd[2] = sdz;
                            __syncwarp();
                            continue;
                        }
                        const int j = jb + lane;
                        bool keep = false;
                        const float4 pj = pn;
                        if (j + 32 < je) pn = __ldg(pos + j + 32);
                        if (j < je) {
                            float ex = tcx - (MODE == kDiffExact ? __fsub_rn(pj.x, jsx) : pj.x);
                            float ey = tcy - (MODE == kDiffExact ? __fsub_rn(pj.y, jsy) : pj.y);
                            float ez = tcz - (MODE == kDiffExact ? __fsub_rn(pj.z, jsz) : pj.z);
                            if (MODE == kDiffWrap) {   /* the centre's minimum image */
                                ex = wrap_d(ex, g.L[0], g.h[0]); ey = wrap_d(ey, g.L[1], g.h[1]); ez = wrap_d(ez, g.L[2], g.h[2]);
                            }
                            const float gx = fmaxf(fabsf(ex) - thx, 0.0f);
                            const float gy = fmaxf(fabsf(ey) - thy, 0.0f);
                            const float gz = fmaxf(fabsf(ez) - thz, 0.0f);
                            keep = gx * gx + gy * gy + gz * gz <= g.rc2;
                        }
                        const unsigned bal = __ballot_sync(0xffffffffu, keep);
                        if (keep) s.idx[cnt + __popc(bal & below)] = j;
                        cnt += __popc(bal);
                        jb += 32;
                    }
                    if (cnt == 0) break;
                    __syncwarp();
                    s.jb = jb; s.je = je; s.total = cnt;
                }

                /* ---- 2: which groups each listed particle is within reach of: a lane keeps the mask of
                 * entry 32 b + lane in byte b of (mlo, mhi) ---- */
                __syncwarp();
                unsigned mlo = 0, mhi = 0;
                {
                    const float jsx = s.js[0], jsy = s.js[1], jsz = s.js[2];
                    for (int e0 = 0; e0 < cnt; e0 += 32) {
                        const int e = e0 + lane;
                        unsigned m = 0;
                        if (e < cnt) {
                            const float4 pj = __ldg(pos + s.idx[e]);
                            float xj = pj.x, yj = pj.y, zj = pj.z;
                            if (MODE == kDiffExact) { xj = __fsub_rn(xj, jsx); yj = __fsub_rn(yj, jsy); zj = __fsub_rn(zj, jsz); }
                            s.fj[0][e] = 0.0f; s.fj[1][e] = 0.0f; s.fj[2][e] = 0.0f;
                            if (EXTRA) s.cj[e] = 0;
#pragma unroll
                            for (int k = 0; k < kTileGroups; ++k) {
                                if (k == kTileGroups / 2 && s.ngr <= kTileGroups / 2) break;
                                const float4 gc = s.g[k][0], gh = s.g[k][1];
                                float ex = gc.x - xj, ey = gc.y - yj, ez = gc.z - zj;
                                if (MODE == kDiffWrap) {
                                    ex = wrap_d(ex, g.L[0], g.h[0]); ey = wrap_d(ey, g.L[1], g.h[1]); ez = wrap_d(ez, g.L[2], g.h[2]);
                                }
                                const float gx = fmaxf(fabsf(ex) - gh.x, 0.0f);
                                const float gy = fmaxf(fabsf(ey) - gh.y, 0.0f);
                                const float gz = fmaxf(fabsf(ez) - gh.z, 0.0f);
                                if (gx * gx + gy * gy + gz * gz <= g.rc2) m |= 1u << k;
                            }
                        }
                        if (e0 < 128) mlo |= m << (e0 >> 2); else mhi |= m << ((e0 - 128) >> 2);
                    }
                }
                __syncwarp();

                /* ---- 3: the pairs, group by group.  In the home cell's own column a pair is counted
                 * once (i < j) and two particles may coincide; elsewhere neither can happen ---- */
                auto pairs = [&](auto own) {
                    constexpr bool SELF = decltype(own)::value;
                    for (int gi = FINE ? warp : 0; gi < s.ngr; gi += FINE ? kWarpsPerCta : 1) {
                        /* the group's list: the tile-list entries with its bit, in order */
                        int len = 0;
                        {
                            const unsigned wlo = mlo >> gi, whi = mhi >> gi;
#pragma unroll
                            for (int bk = 0; bk < kListBlocks; ++bk) {
                                if (bk == 4 && s.total <= 128) break;
                                const bool in = (bk < 4 ? wlo >> (8 * bk) : whi >> (8 * (bk - 4))) & 1u;
                                const unsigned bal = __ballot_sync(0xffffffffu, in);
                                if (in) s.list[len + __popc(bal & below)] = (unsigned char)(32 * bk + lane);
                                len += __popc(bal);
                            }
                        }
                        if (len == 0) continue;
                        __syncwarp();
                        float xi[4], yi[4], zi[4], qi[4];
                        int tti[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float4 p = s.i[4 * gi + k];
                            xi[k] = p.x; yi[k] = p.y; zi[k] = p.z; qi[k] = p.w;
                            tti[k] = s.it[4 * gi + k];
                        }
                        const int ig = s.i0 + 4 * gi;
                        const float jsx = s.js[0], jsy = s.js[1], jsz = s.js[2];
                        const float sdx = s.sd[0], sdy = s.sd[1], sdz = s.sd[2];
                        float fi[12];
#pragma unroll
                        for (int t = 0; t < 12; ++t) fi[t] = 0.0f;
                        int ci[4] = {0, 0, 0, 0};
                        float acc_elj = 0.0f, acc_ec = 0.0f, acc_vir = 0.0f;
                        for (int c0 = 0; c0 < len; c0 += 32) {
                            float xj = -far, yj = -far, zj = -far, qj = 0.0f;
                            int ttj = 0, e = -1, j = 0;
                            if (c0 + lane < len) {
                                e = s.list[c0 + lane];
                                j = s.idx[e];
                                const float4 pj = __ldg(pos + j);
                                xj = pj.x; yj = pj.y; zj = pj.z; qj = pj.w;
                                if (MODE == kDiffExact) { xj = __fsub_rn(xj, jsx); yj = __fsub_rn(yj, jsy); zj = __fsub_rn(zj, jsz); }
                                ttj = __ldg(ptype + j);
                            }
                            float fjx = 0.0f, fjy = 0.0f, fjz = 0.0f;
                            int cj = 0;
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const float dx = pair_diff<MODE>(xi[k], xj, g.L[0], g.h[0], sdx);
                                const float dy = pair_diff<MODE>(yi[k], yj, g.L[1], g.h[1], sdy);
                                const float dz = pair_diff<MODE>(zi[k], zj, g.L[2], g.h[2], sdz);
                                const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                                bool ok = r2 <= g.rc2;
                                if (SELF) ok = ok && r2 > 0.0f && ig + k < j;
                                const float r2e = ORDER == 0 ? (ok ? r2 : g.rc2) : fmaxf(r2, tab.r2min);
                                float v14 = 0.0f, v8 = 0.0f, v3 = 0.0f, v12 = 0.0f, v6 = 0.0f, v1 = 0.0f;
                                pair_functions_if<ORDER, SEP, EXTRA, COUL>(tab, r2e, ok, v14, v8, v3, v12, v6, v1);
                                const float2 pf = sCoefF[tti[k] + ttj];
                                const float qq = __fmul_rn(qi[k], qj);
                                float fs = combine_force<SEP>(make_float4(pf.x, pf.y, 0.0f, 0.0f), qq, COUL, v14, v8, v3);
                                fs = ok ? fs : 0.0f;
                                if (SEP) {
                                    const float fx = __fmul_rn(fs, dx), fy = __fmul_rn(fs, dy), fz = __fmul_rn(fs, dz);
                                    fi[3 * k] += fx; fi[3 * k + 1] += fy; fi[3 * k + 2] += fz;
                                    fjx -= fx; fjy -= fy; fjz -= fz;
                                } else {
                                    fi[3 * k] = __fmaf_rn(fs, dx, fi[3 * k]);
                                    fi[3 * k + 1] = __fmaf_rn(fs, dy, fi[3 * k + 1]);
                                    fi[3 * k + 2] = __fmaf_rn(fs, dz, fi[3 * k + 2]);
                                    fjx = __fmaf_rn(-fs, dx, fjx);
                                    fjy = __fmaf_rn(-fs, dy, fjy);
                                    fjz = __fmaf_rn(-fs, dz, fjz);
                                }
                                acc_pairs += ok ? 1u : 0u;
                                if (EXTRA) {
                                    ci[k] += ok ? 1 : 0;
                                    cj += ok ? 1 : 0;
                                    acc_below += (ORDER > 0 && ok && r2 < tab.r2min) ? 1u : 0u;
                                    const float2 pe = sCoefE[tti[k] + ttj];
                                    const float el = combine_elj<SEP>(make_float4(0.0f, 0.0f, pe.x, pe.y), v12, v6);
                                    acc_elj += ok ? el : 0.0f;
                                    if (COUL) acc_ec += ok ? __fmul_rn(qq, v1) : 0.0f;
                                    acc_vir += ok ? __fmul_rn(fs, r2) : 0.0f;
                                }
                            }
                            if (e >= 0) {
                                s.fj[0][e] += fjx; s.fj[1][e] += fjy; s.fj[2][e] += fjz;
                                if (EXTRA) s.cj[e] += cj;
                            }
                        }
                        reduce_scatter12(fi, lane);
                        {   /* to the global sums: lane 8 k + 2 c, component c of particle k */
                            const int k = ig + (lane >> 3), c = (lane & 7) >> 1;
                            if ((lane & 1) == 0 && c < 3 && k < s.i1 && fi[0] != 0.0f) {
                                if (!(fabsf(fi[0]) < kFixMax) && err) atomicOr(err, kErrForce);
                                atomicAdd(F64 + (size_t)c * n + k, to_fixed(fi[0]));
                            }
                        }
                        if (EXTRA) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const int c = __reduce_add_sync(0xffffffffu, ci[k]);
                                if (lane == 0) s.ci[4 * gi + k] += c;
                            }
                            float e;
                            ehi[0] = two_sum(ehi[0], acc_elj, e); elo[0] += e;
                            if (COUL) { ehi[1] = two_sum(ehi[1], acc_ec, e); elo[1] += e; }
                            ehi[2] = two_sum(ehi[2], acc_vir, e); elo[2] += e;
                        }
                        __syncwarp();   /* the next group's lanes hold other entries of the list */
                    }
                };
                if (s.self) pairs(std::true_type{});
                else pairs(std::false_type{});
                /* ---- 4: the list's j forces: one atomic per particle and component that received a
                 * pair.  Warps that share the item add their sums in group order, the order in which
                 * one warp would have added them ---- */
                if (FINE) __syncthreads();
                for (int e = FINE ? (int)threadIdx.x : lane; e < s.total; e += FINE ? 32 * kWarpsPerCta : 32) {
                    float v0 = s.fj[0][e], v1 = s.fj[1][e], v2 = s.fj[2][e];
                    int cj = EXTRA ? s.cj[e] : 0;
                    if (FINE) {
                        v0 = v1 = v2 = 0.0f;
                        cj = 0;
#pragma unroll
                        for (int w = 0; w < kWarpsPerCta; ++w) {
                            v0 += all[w].fj[0][e]; v1 += all[w].fj[1][e]; v2 += all[w].fj[2][e];
                            if (EXTRA) cj += all[w].cj[e];
                        }
                    }
                    const int j = s.idx[e];
                    if (v0 != 0.0f || v1 != 0.0f || v2 != 0.0f) flush_force<0>(F64, nullptr, n, j, v0, v1, v2, err);
                    if (EXTRA && cj) atomicAdd(counts + j, cj);
                }
                if (FINE) __syncthreads();
                __syncwarp();
            }
            if (EXTRA && s.i0 + lane < s.i1 && (!FINE || (lane >> 2) == warp) && s.ci[lane])
                atomicAdd(counts + s.i0 + lane, s.ci[lane]);
            __syncwarp();
        }

        unsigned c1 = __reduce_add_sync(0xffffffffu, acc_pairs);
        unsigned c2 = EXTRA ? __reduce_add_sync(0xffffffffu, acc_below) : 0u;
        double e1 = 0.0, e2 = 0.0, e3 = 0.0;
        if (EXTRA) {
            e1 = hi_lo(ehi[0], elo[0]); e2 = COUL ? hi_lo(ehi[1], elo[1]) : 0.0; e3 = hi_lo(ehi[2], elo[2]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                e1 += __shfl_xor_sync(0xffffffffu, e1, o);
                if (COUL) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
                e3 += __shfl_xor_sync(0xffffffffu, e3, o);
            }
        }
        if (FINE) {
            if (lane == 0) {
                s.pairs = c1; s.below = c2;
                if (EXTRA) { s.e[0] = e1; s.e[1] = e2; s.e[2] = e3; }
            }
            __syncthreads();
            if (warp != 0) continue;
            for (int w = 1; w < kWarpsPerCta; ++w) {
                c1 += all[w].pairs; c2 += all[w].below;
                if (EXTRA) { e1 += all[w].e[0]; e2 += all[w].e[1]; e3 += all[w].e[2]; }
            }
        }
        if (lane == 0) {
            UnitOut u;
            u.e_lj = e1; u.e_coul = e2; u.virial = e3;
            u.pairs = c1; u.below = c2;
            uout[b] = u;
            pairs_sum += c1;
        }
    }
    if (lane == 0) add_pairs(tot, pairs_sum);
}

/* One set: every order x extra x Coulomb x fine (x arithmetic mode for the reference's difference
 * rules; the exact rule is instantiated with fused arithmetic only).  MODE kDiffShift and kDiffExact:
 * one system; BATCH: half-shell replicas (kDiffShift), and replicas with fewer than 3 cells per axis
 * but every edge above 2 rc (kDiffWrap). */
template <int MODE, bool BATCH>
list_fn pick_force_list(int order, bool sep, bool extra, bool coul, bool fine) {
    auto w = [&](auto ord, auto sp, auto ex) -> list_fn {
        constexpr int O = decltype(ord)::value;
        constexpr bool S = decltype(sp)::value, E = decltype(ex)::value;
        if (fine)
            return coul ? (list_fn)k_force_list<O, S, E, MODE, true, true, BATCH>
                        : (list_fn)k_force_list<O, S, E, MODE, false, true, BATCH>;
        return coul ? (list_fn)k_force_list<O, S, E, MODE, true, false, BATCH>
                    : (list_fn)k_force_list<O, S, E, MODE, false, false, BATCH>;
    };
    auto se = [&](auto ord) -> list_fn {
        using T = std::true_type;
        using F = std::false_type;
        if (MODE != kDiffExact && sep) return extra ? w(ord, T{}, T{}) : w(ord, T{}, F{});
        return extra ? w(ord, F{}, T{}) : w(ord, F{}, F{});
    };
    switch (order) {
        case 0: return se(std::integral_constant<int, 0>{});
        case 1: return se(std::integral_constant<int, 1>{});
        case 2: return se(std::integral_constant<int, 2>{});
        default: return se(std::integral_constant<int, 3>{});
    }
}

extern template list_fn pick_force_list<kDiffShift, false>(int, bool, bool, bool, bool);
extern template list_fn pick_force_list<kDiffExact, false>(int, bool, bool, bool, bool);
extern template list_fn pick_force_list<kDiffShift, true>(int, bool, bool, bool, bool);
extern template list_fn pick_force_list<kDiffWrap, true>(int, bool, bool, bool, bool);

}  // namespace mdrl
