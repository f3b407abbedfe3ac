/*
 * mdrl_cmodel.cu — the drop-in for the reference C model, int MD_Evaluation_Model()
 * (Range_Limited/C_Model_ForceEval/MD_Evaluation_Model.h:1, .cpp:9-205), on the GPU.
 *
 * The reference runs an all-pairs O(N^2) FP32 LJ force with minimum-image PBC, a symplectic
 * Euler update and prints the energies of every iteration.  This file keeps its constants and
 * its rounding: every float expression is evaluated in the reference's types and order with
 * separately rounded intrinsics, and pow(float, int) -- which C++ evaluates in double and the
 * reference stores to float -- is the correctly rounded double power (exact products and a
 * double-double product for the 6th and 7th powers) converted to float.  Each reference
 * particle's force is summed over j in index order, and the energies are summed over i in index
 * order, so the printed values match the reference line for line.
 *
 * One launch per iteration.  A CTA owns a particle: its threads test the j's (moving each from the
 * previous iteration's position on the way, so no launch of its own moves the particles), compact
 * the ones within the cutoff in j order and evaluate those in parallel; only the additions are
 * serial, one lane per component over the compacted values (adding nothing for a rejected j is what
 * the reference does).  One more CTA sums the previous iteration's energies meanwhile.
 * What bounded the form with a thread per particle (500 atoms: 787 us per iteration, 80 ms for 100):
 * 4 CTAs on 152 SMs, and FP64, which this part runs at 1/64 of its FP32 rate, in every step of a
 * 500-long serial loop.  The minimum image needs no FP64 (cmin_image), and the powers are taken for
 * compacted pairs only.
 */
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "mdrl_internal.h"

using namespace mdrl;

namespace {

struct CConst {
    float eps, sig12, sig6, mass, dt, rc2, box;
};

struct DD { double h, l; };

__device__ __forceinline__ DD two_prod(double a, double b) {
    const double p = __dmul_rn(a, b);
    return {p, __fma_rn(a, b, -p)};
}

__device__ __forceinline__ DD dd_mul(DD a, DD b) {
    const double p = __dmul_rn(a.h, b.h);
    double e = __fma_rn(a.h, b.h, -p);
    e = __fma_rn(a.h, b.l, e);
    e = __fma_rn(a.l, b.h, e);
    const double s = __dadd_rn(p, e);
    return {s, __dsub_rn(e, __dsub_rn(s, p))};
}

/* (float)pow((double)x, k) for k = 3, 4, 6, 7 with x a float. */
__device__ __forceinline__ void cpow(float xf, float &p3, float &p4, float &p6, float &p7) {
    const double x = (double)xf;
    const double x2 = __dmul_rn(x, x);         /* exact: 48 significant bits */
    const DD x3 = two_prod(x2, x);              /* exact */
    const DD x4 = two_prod(x2, x2);             /* exact */
    const DD x6 = dd_mul(x3, x3);
    const DD x7 = dd_mul(x4, x3);
    p3 = __double2float_rn(x3.h);
    p4 = __double2float_rn(x4.h);
    p6 = __double2float_rn(__dadd_rn(x6.h, x6.l));
    p7 = __double2float_rn(__dadd_rn(x7.h, x7.l));
}

/* dx -= L * (int)(dx/L +- 0.5)  (MD_Evaluation_Model.cpp:81-98).  The reference adds 0.5 in double,
 * which is exact, and truncates: |dx/L| rounded half up.  With f = floor(|dx/L|), |dx/L| - f is exact
 * in FP32, so comparing it with 0.5 decides the same way. */
__device__ __forceinline__ float cmin_image(float d, float L) {
    const float q = fabsf(__fdiv_rn(d, L)), f = floorf(q);
    const float k = fminf(f + (__fsub_rn(q, f) >= 0.5f ? 1.0f : 0.0f), 2147483648.0f);   /* an int, as there */
    return __fsub_rn(d, __fmul_rn(L, d >= 0.0f ? k : -k));
}

/* x += v dt with one wrap into [0, L) (.cpp:164-202). */
__device__ __forceinline__ float cmove(float x, float v, const CConst &k) {
    float p = __fadd_rn(x, __fmul_rn(v, k.dt));
    if (p < 0.0f) p = __fadd_rn(p, k.box);
    else if (p >= k.box) p = __fsub_rn(p, k.box);
    return p;
}

constexpr int kCmThreads = 128;
constexpr int kCmList = 512;     /* compacted pairs evaluated at a time */

/* System energies of one iteration, summed over i in order (.cpp:152-158): lane 0 the potential, lane 1
 * the kinetic energy, from values staged in shared memory. */
__device__ __forceinline__ void cm_energy(int n, const float *__restrict__ ev, const float *__restrict__ ek,
                                          float *__restrict__ out, float (*s)[kCmList]) {
    float sum = 0.0f;
    for (int i0 = 0; i0 < n; i0 += kCmList) {
        const int m = min(kCmList, n - i0);
        __syncthreads();
        for (int t = threadIdx.x; t < m; t += kCmThreads) { s[0][t] = ev[i0 + t]; s[1][t] = ek[i0 + t]; }
        __syncthreads();
        if (threadIdx.x < 2) {
            const float *v = s[threadIdx.x];
#pragma unroll 8
            for (int t = 0; t < m; ++t) sum = __fadd_rn(sum, v[t]);
        }
    }
    if (threadIdx.x == 0) out[0] = __double2float_rn(__dmul_rn((double)sum, 0.5));
    if (threadIdx.x == 1) out[1] = sum;
}

/* One iteration (.cpp:57-158) from the previous one's positions and velocities (move: they are moved
 * first).  CTA i < n: force, energy and velocity update of particle i; CTA n (when eout is given): the
 * previous iteration's energies. */
__global__ void __launch_bounds__(kCmThreads)
k_cm_step(int n, int move, const float *__restrict__ pos0, const float *__restrict__ vel0, float *__restrict__ pos1,
          float *__restrict__ vel1, const float *__restrict__ ev0, const float *__restrict__ ek0,
          float *__restrict__ ev1, float *__restrict__ ek1, float *__restrict__ eout, int *__restrict__ counts,
          CConst k) {
    __shared__ float s_v[4][kCmList];        /* dx, dy, dz, r2 of the pairs, then Fx, Fy, Fz, E */
    __shared__ int s_warp[kCmThreads / 32];
    __shared__ float s_sum[4];
    if ((int)blockIdx.x == n) {
        cm_energy(n, ev0, ek0, eout, s_v);
        return;
    }
    const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float r[3], v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        v[d] = vel0[3 * i + d];
        r[d] = move ? cmove(pos0[3 * i + d], v[d], k) : pos0[3 * i + d];
    }
    const float e4 = __fmul_rn(4.0f, k.eps), e48 = __fmul_rn(48.0f, k.eps), e24 = __fmul_rn(24.0f, k.eps);
    const float c12 = __fmul_rn(e4, k.sig12), c6 = __fmul_rn(e4, k.sig6);
    const float c14 = __fmul_rn(e48, k.sig12), c8 = __fmul_rn(e24, k.sig6);
    float sum = 0.0f;                        /* lane c < 4 of warp 0: component c */
    int cnt = 0, nb = 0;
    for (int j0 = 0; j0 < n; j0 += kCmThreads) {
        const int j = j0 + tid;
        float d[3] = {0.0f, 0.0f, 0.0f}, r2 = 0.0f;
        if (j < n) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float x = move ? cmove(pos0[3 * j + c], vel0[3 * j + c], k) : pos0[3 * j + c];
                d[c] = cmin_image(__fsub_rn(r[c], x), k.box);
            }
            r2 = __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])), __fmul_rn(d[2], d[2]));
        }
        const bool ok = r2 > 0.0f && r2 <= k.rc2;
        const unsigned bal = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) s_warp[warp] = __popc(bal);
        __syncthreads();
        int at = cnt + __popc(bal & ((1u << lane) - 1u)), tot = 0;
#pragma unroll
        for (int w = 0; w < kCmThreads / 32; ++w) {
            if (w < warp) at += s_warp[w];
            tot += s_warp[w];
        }
        if (ok) { s_v[0][at] = d[0]; s_v[1][at] = d[1]; s_v[2][at] = d[2]; s_v[3][at] = r2; }
        cnt += tot;
        nb += tot;
        __syncthreads();
        if (cnt <= kCmList - kCmThreads && j0 + kCmThreads < n) continue;
        for (int e = tid; e < cnt; e += kCmThreads) {
            const float inv_r2 = __fdiv_rn(1.0f, s_v[3][e]);
            float p3, p4, p6, p7;
            cpow(inv_r2, p3, p4, p6, p7);
            const float vdw12 = __fmul_rn(c12, p6), vdw6 = __fmul_rn(c6, p3);
            const float vdw14 = __fmul_rn(c14, p7), vdw8 = __fmul_rn(c8, p4);
            const float Fv = __fsub_rn(vdw14, vdw8);
            s_v[0][e] = __fmul_rn(Fv, s_v[0][e]);
            s_v[1][e] = __fmul_rn(Fv, s_v[1][e]);
            s_v[2][e] = __fmul_rn(Fv, s_v[2][e]);
            s_v[3][e] = __fsub_rn(vdw12, vdw6);
        }
        __syncthreads();
        if (tid < 4) {
            const float *a = s_v[tid];
#pragma unroll 8
            for (int e = 0; e < cnt; ++e) sum = __fadd_rn(sum, a[e]);
        }
        cnt = 0;
        __syncthreads();
    }
    if (tid < 4) s_sum[tid] = sum;
    __syncthreads();
    if (tid != 0) return;
    ev1[i] = s_sum[3];
    if (counts) counts[i] = nb;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        v[c] = __fadd_rn(v[c], __fmul_rn(__fdiv_rn(s_sum[c], k.mass), k.dt));
        pos1[3 * i + c] = r[c];
        vel1[3 * i + c] = v[c];
    }
    const float v2 = __fadd_rn(__fadd_rn(__fmul_rn(v[0], v[0]), __fmul_rn(v[1], v[1])), __fmul_rn(v[2], v[2]));
    ek1[i] = __double2float_rn(__dmul_rn(__dmul_rn(0.5, (double)k.mass), (double)v2));
}

/* The end of the last iteration: its energies (CTA 0) and the move. */
__global__ void __launch_bounds__(kCmThreads)
k_cm_finish(int n, float *__restrict__ pos, const float *__restrict__ vel, const float *__restrict__ ev,
            const float *__restrict__ ek, float *__restrict__ eout, CConst k) {
    __shared__ float s_v[2][kCmList];
    if (blockIdx.x == 0) {
        cm_energy(n, ev, ek, eout, s_v);
        return;
    }
    const int i = (blockIdx.x - 1) * kCmThreads + threadIdx.x;
    if (i < 3 * n) pos[i] = cmove(pos[i], vel[i], k);
}

struct DevBuf {
    void *p = nullptr;
    ~DevBuf() { if (p) cudaFree(p); }
};

}  // namespace

#define CM_CUDA(call)                                                                    \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess) {                                                         \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));               \
            return MDRL_ERR_CUDA;                                                        \
        }                                                                                \
    } while (0)

extern "C" mdrl_status mdrl_cmodel_run(int n, int iters, float box, float cutoff, float *pos, float *vel,
                                       float *energy, int *counts) {
    if (n <= 0 || iters < 0 || !(box > 0.0f) || !(cutoff > 0.0f) || !pos || !vel || (iters > 0 && !energy)) {
        set_error("mdrl_cmodel_run: invalid argument");
        return MDRL_ERR_INVALID_ARG;
    }
    /* The reference's constants (.cpp:14-24), in its types. */
    CConst k;
    k.eps = (float)(1.995996 * 1.995996);
    const float sigma = (float)(0.1675 * 2);
    k.sig12 = (float)std::pow((double)sigma, 12.0);
    k.sig6 = (float)std::pow((double)sigma, 6.0);
    const float weight = 39.95f, nav = 6.022e23f;
    k.mass = weight / nav / 1000;
    k.dt = (float)2E-15;
    k.rc2 = cutoff * cutoff;
    k.box = box;
    /* one allocation: positions and velocities (two slots each, one per iteration parity), per-particle
     * energies (two slots), the energies of every iteration, counts */
    const size_t m = (size_t)n, b3 = sizeof(float) * 3 * m;
    DevBuf buf;
    CM_CUDA(cudaMalloc(&buf.p, sizeof(float) * (12 * m + 4 * m + 2 * (size_t)(iters > 0 ? iters : 1)) +
                                   (counts ? sizeof(int) * m : 0)));
    float *f = (float *)buf.p;
    float *dpos[2] = {f, f + 3 * m}, *dvel[2] = {f + 6 * m, f + 9 * m};
    float *dev[2] = {f + 12 * m, f + 13 * m}, *dek[2] = {f + 14 * m, f + 15 * m}, *dout = f + 16 * m;
    int *dcnt = counts ? (int *)(dout + 2 * (size_t)(iters > 0 ? iters : 1)) : nullptr;
    CM_CUDA(cudaMemcpy(dpos[0], pos, b3, cudaMemcpyHostToDevice));
    CM_CUDA(cudaMemcpy(dvel[0], vel, b3, cudaMemcpyHostToDevice));
    int a = 0;
    for (int it = 0; it < iters; ++it, a ^= 1)
        k_cm_step<<<n + (it > 0 ? 1 : 0), kCmThreads>>>(n, it > 0, dpos[a], dvel[a], dpos[1 - a], dvel[1 - a], dev[a],
                                                        dek[a], dev[1 - a], dek[1 - a], dout + 2 * (it - 1), dcnt, k);
    if (iters > 0)
        k_cm_finish<<<1 + (3 * n + kCmThreads - 1) / kCmThreads, kCmThreads>>>(n, dpos[a], dvel[a], dev[a], dek[a],
                                                                                dout + 2 * (iters - 1), k);
    CM_CUDA(cudaGetLastError());
    CM_CUDA(cudaDeviceSynchronize());
    CM_CUDA(cudaMemcpy(pos, dpos[a], b3, cudaMemcpyDeviceToHost));
    CM_CUDA(cudaMemcpy(vel, dvel[a], b3, cudaMemcpyDeviceToHost));
    if (iters > 0) CM_CUDA(cudaMemcpy(energy, dout, sizeof(float) * 2 * iters, cudaMemcpyDeviceToHost));
    if (counts && iters > 0) CM_CUDA(cudaMemcpy(counts, dcnt, sizeof(int) * m, cudaMemcpyDeviceToHost));
    return MDRL_OK;
}

/* The reference reads an argon PDB: five header lines, then one atom per line whose 7th-9th
 * whitespace-separated fields are x, y, z (.cpp:38-55). */
extern "C" int MD_Evaluation_Model(void) {
    const char *path = std::getenv("MDRL_INPUT");
    if (!path || !*path) {
        set_error("MD_Evaluation_Model: set MDRL_INPUT to the argon PDB file");
        return 0;
    }
    const char *ns = std::getenv("MDRL_N");
    const char *is = std::getenv("MDRL_ITERS");
    const int n = ns ? std::atoi(ns) : 500;
    const int iters = is ? std::atoi(is) : 100;
    if (n <= 0 || iters < 0) { set_error("MD_Evaluation_Model: bad MDRL_N or MDRL_ITERS"); return 0; }
    FILE *fp = std::fopen(path, "r");
    if (!fp) { set_error(std::string("MD_Evaluation_Model: cannot open ") + path); return 0; }
    std::vector<float> pos(3 * (size_t)n, 0.0f), vel(3 * (size_t)n, 0.0f);
    char line[1024];
    for (int i = 0; i < 5; ++i)
        if (!std::fgets(line, sizeof line, fp)) break;
    int got = 0;
    for (int i = 0; i < n; ++i) {
        if (!std::fgets(line, sizeof line, fp)) break;
        float x, y, z;
        if (std::sscanf(line, "%*s %*s %*s %*s %*s %*s %f %f %f", &x, &y, &z) == 3) {
            pos[3 * i] = x; pos[3 * i + 1] = y; pos[3 * i + 2] = z;
            ++got;
        }
    }
    std::fclose(fp);
    if (got != n) {
        set_error("MD_Evaluation_Model: the PDB holds fewer atoms than MDRL_N");
        return 0;
    }
    std::vector<float> energy(2 * (size_t)(iters > 0 ? iters : 1));
    if (mdrl_cmodel_run(n, iters, 24.0f, 8.0f, pos.data(), vel.data(), energy.data(), nullptr) != MDRL_OK)
        return 0;
    for (int it = 0; it < iters; ++it)
        std::printf("Iteration %d, System energy is %f, Kinetic Energy is %f\n", it, energy[2 * it],
                    energy[2 * it + 1]);
    std::fflush(stdout);
    return 1;
}
