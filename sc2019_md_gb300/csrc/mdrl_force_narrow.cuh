/*
 * mdrl_force_narrow.cuh — the default tile's half-shell units one warp each (sm_103a), for dynamics of
 * systems with few particles per cell.
 *
 * The CTA kernel (mdrl_force.cuh) deals a unit's pieces (32 i x 8 spp j) to 4 warps.  A unit of two
 * cells of 46 particles has 2 pieces and one of 27 has 1, so half or three quarters of its warps only
 * wait at barriers.  Here a warp runs a whole unit, its pieces one after the other, and keeps the 4
 * warps' accumulators apart in its own shared memory (piece p adds to accumulator p mod 4).  Every
 * FP32 sum is formed from the same values in the same order as the CTA kernel forms it: forces and
 * trajectories are its, bit for bit (energies, summed per lane over other pieces, to FP32 rounding).
 * Blocks of 4 i x 8 j whose boxes are beyond rc are skipped (the exact test of mdrl_force_warp.cuh);
 * they add nothing in the CTA kernel either.
 *
 * A cell above kNarrowCell particles takes its accumulators from global scratch in the CTA kernel's
 * chunks of 256: slow, and what keeps the path right whatever the particles do.
 *
 * Latency-bound, as the CTA kernel, with 16 working warps per SM instead of 4 to 8.  A launch by CTAs
 * and here: 24,000 atoms at 14 per cell 172 -> 73 us, at 33 120 -> 61; 90,000 at 33 421 -> 192, at 68
 * 329 -> 227; 1,728 at 27 20 -> 16.  Accumulators of 64 particles run 33 per cell 3 to 7 % faster and
 * 68 per cell 1.6 times slower, of 128 10 % slower and 4 % faster; 12 CTAs per SM instead of 16
 * 13 % slower at 33, 20 and 24 never faster.
 */
#pragma once

#include "mdrl_force_warp.cuh"

namespace mdrl {

constexpr int kNarrowCell = 96;                 /* particles per cell the shared accumulators hold */
constexpr int kNarrowCtas = 16;                 /* CTAs (warps) per SM: more would spill, fewer wait longer */
constexpr int kNarrowWarps = 4;                 /* the emulated CTA's warps */
constexpr size_t kNarrowScratch = (size_t)kNarrowWarps * 6 * kChunk;   /* floats of scratch per warp */

inline size_t force_narrow_smem_bytes(int ntypes, bool extra) {
    const size_t t2 = (size_t)((ntypes * ntypes + 1) & ~1);
    return sizeof(float2) * t2 * (extra ? 2 : 1) + sizeof(float4) * (2 * 32 + 2 * 8) +
           sizeof(float) * kNarrowWarps * 6 * kNarrowCell;
}

typedef void (*narrow_fn)(const float4 *, const int *, const int *, Geom, TableDev, const float4 *, int, float, int,
                          unsigned long long *, int *, UnitOut *, int, unsigned *, int, int *, int, float *, DevTotals *);

template <int ORDER, bool SEP, bool EXTRA, int MODE, bool COUL>
__global__ void __launch_bounds__(32, kNarrowCtas)
k_force_narrow(const float4 *__restrict__ pos, const int *__restrict__ ptype, const int *__restrict__ cstart, Geom g,
               TableDev tab, const float4 *__restrict__ pcoef, int ntypes, float ke, int n,
               unsigned long long *__restrict__ F64, int *__restrict__ counts, UnitOut *__restrict__ uout, int spp,
               unsigned *__restrict__ err, int unit0, int *__restrict__ work, int nitems, float *__restrict__ scratch,
               DevTotals *tot) {
    const int t2 = (ntypes * ntypes + 1) & ~1;
    extern __shared__ float4 wsm[];
    float2 *sCoefF = reinterpret_cast<float2 *>(wsm);           /* (A14, B8) [T^2] */
    float2 *sCoefE = sCoefF + t2;                               /* (A12, B6) [T^2], EXTRA only */
    float4 *sSB = reinterpret_cast<float4 *>(sCoefE + (EXTRA ? t2 : 0));   /* step boxes [2][32] */
    float4 *sGB = sSB + 2 * 32;                                 /* group boxes of the tile [2][8] */
    float *sAcc = reinterpret_cast<float *>(sGB + 2 * 8);       /* [4][i, j][3][kNarrowCell] */
    const int lane = threadIdx.x, row = lane >> 3, col = lane & 7;
    const float far = 1.0e18f;
    for (int t = lane; t < ntypes * ntypes; t += 32) {
        const float4 c4 = pcoef[t];
        sCoefF[t] = make_float2(c4.x, c4.y);
        if (EXTRA) sCoefE[t] = make_float2(c4.z, c4.w);
    }
    __syncwarp();
    const float margin = 9.5367431640625e-07f * fmaxf(g.L[0], fmaxf(g.L[1], g.L[2]));
    unsigned long long pairs_sum = 0;

    for (;;) {
        int b = 0;
        if (lane == 0) b = atomicAdd(work, 1);
        b = __shfl_sync(0xffffffffu, b, 0);
        if (b >= nitems) break;
        /* unit class position first (self, faces, edges, corners), then home cell */
        const int nh = nitems / kHalfShellCells;
        const int f = c_unit_order[b / nh], h = unit0 / kHalfShellCells + b % nh;
        const int nyz = g.nc[1] * g.nc[2];
        const int hx = h / nyz, hy = (h / g.nc[2]) % g.nc[1], hz = h % g.nc[2];
        int cx = hx + c_halfshell[f][0], cy = hy + c_halfshell[f][1], cz = hz + c_halfshell[f][2];
        const float sx = cx >= g.nc[0] ? -g.L[0] : (cx < 0 ? g.L[0] : 0.0f);
        const float sy = cy >= g.nc[1] ? -g.L[1] : (cy < 0 ? g.L[1] : 0.0f);
        const float sz = cz >= g.nc[2] ? -g.L[2] : (cz < 0 ? g.L[2] : 0.0f);
        cx = cx < 0 ? cx + g.nc[0] : (cx >= g.nc[0] ? cx - g.nc[0] : cx);
        cy = cy < 0 ? cy + g.nc[1] : (cy >= g.nc[1] ? cy - g.nc[1] : cy);
        cz = cz < 0 ? cz + g.nc[2] : (cz >= g.nc[2] ? cz - g.nc[2] : cz);
        const int c = (cx * g.nc[1] + cy) * g.nc[2] + cz;
        const bool self = f == 0;
        const int hs = cstart[h], ni_all = cstart[h + 1] - hs;
        const int cs = cstart[c], nj_all = cstart[c + 1] - cs;
        const bool skip = ni_all > kMaxCellOcc || nj_all > kMaxCellOcc;
        /* exact rule: the box edge comes off the high side's coordinates (see pair_diff) */
        const bool ex = MODE == kDiffExact;
        const float ix = ex ? fminf(sx, 0.0f) : 0.0f, iy = ex ? fminf(sy, 0.0f) : 0.0f, iz = ex ? fminf(sz, 0.0f) : 0.0f;
        const float jx = ex ? fmaxf(sx, 0.0f) : 0.0f, jy = ex ? fmaxf(sy, 0.0f) : 0.0f, jz = ex ? fmaxf(sz, 0.0f) : 0.0f;
        auto ipos = [&](int k) {
            float4 p = __ldg(pos + k);
            if (ex) { p.x = __fadd_rn(p.x, ix); p.y = __fadd_rn(p.y, iy); p.z = __fadd_rn(p.z, iz); }
            return p;
        };
        auto jpos = [&](int k) {
            float4 p = __ldg(pos + k);
            if (ex) { p.x = __fsub_rn(p.x, jx); p.y = __fsub_rn(p.y, jy); p.z = __fsub_rn(p.z, jz); }
            return p;
        };
        float acc_elj = 0.0f, acc_ec = 0.0f, acc_vir = 0.0f;
        unsigned acc_pairs = 0, acc_below = 0;

        /* one chunk pair: particles [i0, i0 + ni) of the home cell against [j0, j0 + nj) of the
         * neighbour; acc: [4][2][3][CAP] */
        auto chunk = [&](float *acc, auto cap, int i0, int ni, int j0, int nj) {
            constexpr int CAP = decltype(cap)::value;
            const bool diag = self && i0 == j0;
            const int nti = (ni + 31) >> 5, S = (nj + 7) >> 3;
            int np = 0;
            for (int ti = 0; ti < nti; ++ti) np += (S - (diag ? 4 * ti : 0) + spp - 1) / spp;
            const int nw = min(np, kNarrowWarps);
            for (int w = 0; w < nw; ++w)
                for (int d = 0; d < 3; ++d) {
                    for (int t = lane; t < ni; t += 32) acc[(w * 6 + d) * CAP + t] = 0.0f;
                    for (int t = lane; t < nj; t += 32) acc[(w * 6 + 3 + d) * CAP + t] = 0.0f;
                }
            if (lane < S) {
                float lx = 3.0e38f, ly = 3.0e38f, lz = 3.0e38f, ux = -3.0e38f, uy = -3.0e38f, uz = -3.0e38f;
                for (int u = 0; u < 8 && 8 * lane + u < nj; ++u) {
                    const float4 pp = jpos(cs + j0 + 8 * lane + u);
                    lx = fminf(lx, pp.x); ly = fminf(ly, pp.y); lz = fminf(lz, pp.z);
                    ux = fmaxf(ux, pp.x); uy = fmaxf(uy, pp.y); uz = fmaxf(uz, pp.z);
                }
                sSB[lane] = make_float4(0.5f * (lx + ux), 0.5f * (ly + uy), 0.5f * (lz + uz), 0.0f);
                sSB[32 + lane] = make_float4(0.5f * (ux - lx), 0.5f * (uy - ly), 0.5f * (uz - lz), 0.0f);
            }
            int p0 = 0;                         /* pieces before this tile's */
            for (int ti = 0; ti < nti; ++ti) {
                const int ib = hs + i0 + ti * 32, im = min(32, ni - ti * 32);
                __syncwarp();
                if (lane < 8) {
                    float lx = 3.0e38f, ly = 3.0e38f, lz = 3.0e38f, ux = -3.0e38f, uy = -3.0e38f, uz = -3.0e38f;
                    for (int r = 0; r < 4 && 4 * lane + r < im; ++r) {
                        const float4 pp = ipos(ib + 4 * lane + r);
                        lx = fminf(lx, pp.x); ly = fminf(ly, pp.y); lz = fminf(lz, pp.z);
                        ux = fmaxf(ux, pp.x); uy = fmaxf(uy, pp.y); uz = fmaxf(uz, pp.z);
                    }
                    const bool some = lx <= ux, sh = MODE == kDiffShift;   /* the unit's shift folds into the centre */
                    sGB[lane] = make_float4(0.5f * (lx + ux) + (sh ? sx : 0.0f), 0.5f * (ly + uy) + (sh ? sy : 0.0f),
                                            0.5f * (lz + uz) + (sh ? sz : 0.0f), 0.0f);
                    sGB[8 + lane] = make_float4(some ? 0.5f * (ux - lx) + margin : -1.0f, 0.5f * (uy - ly) + margin,
                                                0.5f * (uz - lz) + margin, 0.0f);
                }
                __syncwarp();
                unsigned km = 0;                /* live groups of this lane's step */
                if (lane < S) {
                    const float4 jc = sSB[lane], jh = sSB[32 + lane];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float4 tc = sGB[k], th = sGB[8 + k];
                        const float gx = fmaxf(fabsf(tc.x - jc.x) - (th.x + jh.x), 0.0f);
                        const float gy = fmaxf(fabsf(tc.y - jc.y) - (th.y + jh.y), 0.0f);
                        const float gz = fmaxf(fabsf(tc.z - jc.z) - (th.z + jh.z), 0.0f);
                        if (th.x >= 0.0f && gx * gx + gy * gy + gz * gz <= g.rc2) km |= 1u << k;
                    }
                }
                const unsigned alive = __ballot_sync(0xffffffffu, km != 0);
                const int base = diag ? 4 * ti : 0, nst = S - base;
                float xi[8], yi[8], zi[8], qi[8];
                int tti[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int il = row + 4 * k;
                    if (il < im) {
                        const float4 pp = ipos(ib + il);
                        xi[k] = pp.x; yi[k] = pp.y; zi[k] = pp.z;
                        qi[k] = __fmul_rn(ke, pp.w);
                        tti[k] = __ldg(ptype + ib + il) * ntypes;
                    } else {
                        xi[k] = far; yi[k] = far; zi[k] = far; qi[k] = 0.0f; tti[k] = 0;
                    }
                }
                const int tp = (nst + spp - 1) / spp;
                for (int r = 0; r < tp; ++r) {
                    /* the live steps of piece p0 + r */
                    const int k0 = base + r * spp, k1 = min(S, k0 + spp);
                    unsigned todo = alive & (k1 >= 32 ? 0xffffffffu : (1u << k1) - 1u) & ~((1u << k0) - 1u);
                    if (!todo) continue;
                    float *aw = acc + ((p0 + r) % kNarrowWarps) * 6 * CAP;
                    float fi[24];
#pragma unroll
                    for (int t = 0; t < 24; ++t) fi[t] = 0.0f;
                    int ci[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    bool piece_hit = false;
                    for (; todo; todo &= todo - 1u) {
                        const int st = __ffs(todo) - 1;
                        const unsigned live = __shfl_sync(0xffffffffu, km, st);
                        const int jl = 8 * st + col;
                        float xj = -far, yj = -far, zj = -far, qj = 0.0f;
                        int ttj = 0;
                        if (jl < nj) {
                            const float4 pp = jpos(cs + j0 + jl);
                            xj = pp.x; yj = pp.y; zj = pp.z; qj = pp.w;
                            ttj = __ldg(ptype + cs + j0 + jl);
                        }
                        float fjx = 0.f, fjy = 0.f, fjz = 0.f;
                        int cj = 0;
                        bool hit = false;
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            if (!((live >> k) & 1u)) continue;
                            const float dx = pair_diff<MODE>(xi[k], xj, g.L[0], g.h[0], sx);
                            const float dy = pair_diff<MODE>(yi[k], yj, g.L[1], g.h[1], sy);
                            const float dz = pair_diff<MODE>(zi[k], zj, g.L[2], g.h[2], sz);
                            const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                            bool ok = (r2 > 0.0f) && (r2 <= g.rc2);
                            if (diag) ok = ok && (ti * 32 + row + 4 * k < jl);
                            if (ok) {
                                float v14, v8, v3, v12, v6, v1;
                                pair_functions_split<ORDER, SEP, EXTRA>(tab, r2, COUL, v14, v8, v3, v12, v6, v1);
                                const float2 pf = sCoefF[tti[k] + ttj];
                                const float qq = __fmul_rn(qi[k], qj);
                                const float fs = combine_force<SEP>(make_float4(pf.x, pf.y, 0.0f, 0.0f), qq, COUL, v14, v8, v3);
                                const float fx = __fmul_rn(fs, dx), fy = __fmul_rn(fs, dy), fz = __fmul_rn(fs, dz);
                                fi[3 * k] += fx; fi[3 * k + 1] += fy; fi[3 * k + 2] += fz;
                                fjx -= fx; fjy -= fy; fjz -= fz;
                                hit = true;
                                ++acc_pairs;
                                if (EXTRA) {
                                    ++ci[k];
                                    ++cj;
                                    acc_below += (ORDER > 0 && r2 < tab.r2min) ? 1u : 0u;
                                    const float2 pe = sCoefE[tti[k] + ttj];
                                    acc_elj += combine_elj<SEP>(make_float4(0.0f, 0.0f, pe.x, pe.y), v12, v6);
                                    if (COUL) acc_ec += __fmul_rn(qq, v1);
                                    acc_vir += __fmul_rn(fs, r2);
                                }
                            }
                        }
                        if (!__any_sync(0xffffffffu, hit)) continue;
                        piece_hit = true;
#pragma unroll
                        for (int o = 8; o < 32; o <<= 1) {
                            fjx += __shfl_xor_sync(0xffffffffu, fjx, o);
                            fjy += __shfl_xor_sync(0xffffffffu, fjy, o);
                            fjz += __shfl_xor_sync(0xffffffffu, fjz, o);
                            if (EXTRA) cj += __shfl_xor_sync(0xffffffffu, cj, o);
                        }
                        if (jl < nj) {
                            if (row < 3) aw[(3 + row) * CAP + jl] += row == 0 ? fjx : (row == 1 ? fjy : fjz);
                            else if (EXTRA && cj) atomicAdd(counts + cs + j0 + jl, cj);
                        }
                    }
                    if (!piece_hit) continue;
                    reduce_scatter24(fi, col);
                    int cnt_i = 0;
                    if (EXTRA) cnt_i = reduce_scatter8i(ci, col);
                    const int il = ti * 32 + row + 4 * col;
                    if (il < ni) {
                        aw[il] += fi[0];
                        aw[CAP + il] += fi[1];
                        aw[2 * CAP + il] += fi[2];
                        if (EXTRA && cnt_i) atomicAdd(counts + hs + i0 + il, cnt_i);
                    }
                    __syncwarp();
                }
                p0 += tp;
            }
            __syncwarp();
            /* the accumulators summed in warp order, as the CTA kernel sums them */
            for (int t = lane; t < ni; t += 32) {
                float v[3] = {0.0f, 0.0f, 0.0f};
                for (int w = 0; w < nw; ++w)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        v[d] += acc[(w * 6 + d) * CAP + t];
                        if (diag) v[d] += acc[(w * 6 + 3 + d) * CAP + t];
                    }
                if (v[0] != 0.0f || v[1] != 0.0f || v[2] != 0.0f)
                    flush_force<0>(F64, nullptr, n, hs + i0 + t, v[0], v[1], v[2], err);
            }
            if (!diag)
                for (int t = lane; t < nj; t += 32) {
                    float v[3] = {0.0f, 0.0f, 0.0f};
                    for (int w = 0; w < nw; ++w)
#pragma unroll
                        for (int d = 0; d < 3; ++d) v[d] += acc[(w * 6 + 3 + d) * CAP + t];
                    if (v[0] != 0.0f || v[1] != 0.0f || v[2] != 0.0f)
                        flush_force<0>(F64, nullptr, n, cs + j0 + t, v[0], v[1], v[2], err);
                }
            __syncwarp();
        };
        if (!skip) {
            if (ni_all <= kNarrowCell && nj_all <= kNarrowCell) {
                if (ni_all && nj_all) chunk(sAcc, std::integral_constant<int, kNarrowCell>{}, 0, ni_all, 0, nj_all);
            } else {
                for (int i0 = 0; i0 < ni_all; i0 += kChunk)
                    for (int j0 = self ? i0 : 0; j0 < nj_all; j0 += kChunk)
                        chunk(scratch + kNarrowScratch * blockIdx.x, std::integral_constant<int, kChunk>{}, i0,
                              min(kChunk, ni_all - i0), j0, min(kChunk, nj_all - j0));
            }
        }

        const unsigned c1 = __reduce_add_sync(0xffffffffu, acc_pairs);
        unsigned c2 = 0;
        double e1 = 0.0, e2 = 0.0, e3 = 0.0;
        if (EXTRA) {
            c2 = __reduce_add_sync(0xffffffffu, acc_below);
            e1 = acc_elj; e2 = acc_ec; e3 = acc_vir;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                e1 += __shfl_xor_sync(0xffffffffu, e1, o);
                e2 += __shfl_xor_sync(0xffffffffu, e2, o);
                e3 += __shfl_xor_sync(0xffffffffu, e3, o);
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

template <int MODE>
narrow_fn pick_force_narrow(int order, bool sep, bool extra, bool coul) {
    auto w = [&](auto ord, auto sp, auto ex) -> narrow_fn {
        constexpr int O = decltype(ord)::value;
        constexpr bool S = decltype(sp)::value, E = decltype(ex)::value;
        return coul ? (narrow_fn)k_force_narrow<O, S, E, MODE, true> : (narrow_fn)k_force_narrow<O, S, E, MODE, false>;
    };
    auto se = [&](auto ord) -> narrow_fn {
        using T = std::true_type;
        using F = std::false_type;
        if (MODE == kDiffShift && sep) return extra ? w(ord, T{}, T{}) : w(ord, T{}, F{});
        return extra ? w(ord, F{}, T{}) : w(ord, F{}, F{});
    };
    switch (order) {
        case 0: return se(std::integral_constant<int, 0>{});
        case 1: return se(std::integral_constant<int, 1>{});
        case 2: return se(std::integral_constant<int, 2>{});
        default: return se(std::integral_constant<int, 3>{});
    }
}

extern template narrow_fn pick_force_narrow<kDiffShift>(int, bool, bool, bool);
extern template narrow_fn pick_force_narrow<kDiffExact>(int, bool, bool, bool);

}  // namespace mdrl
