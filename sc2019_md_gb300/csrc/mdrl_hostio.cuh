/*
 * mdrl_hostio.cuh — host arrays as kernels read and write them (GB300: the GPU shares the host's page
 * tables over NVLink-C2C, so it can use pageable memory in place).
 *
 * A call's host arrays used to go through one cudaMemcpyAsync each, ~8 us apiece whatever their size
 * (frame of 1,728 atoms: 9 copies, 105 us), and a copy into pages that nobody has touched yet faulted
 * them in one by one from the device side (47 us per 64 KB page: 75 ms for the 104 MB frame of 2.9M
 * atoms, 0.9 ms into touched pages).  Now one kernel moves all arrays of a call (copy_arrays), and the
 * pages of pageable outputs are populated by the host first (populate), in force evaluations while
 * the GPU computes: frame of 1,728 atoms 50 us, of 2.9M atoms 3.4 ms.
 */
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <thread>

#include "mdrl_ctx.cuh"

namespace mdrl {

constexpr int kMaxArrays = 9;
constexpr size_t kPopulateChunk = size_t(8) << 20;   /* bytes per populating thread, at most 8 threads */

/* The device address of p when the context's device can read and write it in place: page-locked
 * host memory (cudaHostAlloc / cudaHostRegister, mapped), managed memory, memory of this device, or
 * pageable memory where the device walks the host's page tables (*pageable is then set); nullptr
 * otherwise (the caller stages through copies).  Kernels access whole elements, so an address that is
 * not a multiple of `align`, in whatever memory, is left to the copies, which take any. */
inline void *device_view(const mdrl_ctx *c, const void *p, size_t align, bool *pageable = nullptr) {
    if ((uintptr_t)p % align) return nullptr;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged) return a.devicePointer;
    if (a.type == cudaMemoryTypeDevice && a.device == c->p.device) return a.devicePointer;
    if (a.type != cudaMemoryTypeUnregistered || !c->host_tables) return nullptr;
    if (pageable) *pageable = true;
    return const_cast<void *>(p);
}

/* Whether [a, a + na) and [b, b + nb) share a byte (null: no array). */
inline bool overlap(const void *a, size_t na, const void *b, size_t nb) {
    const uintptr_t pa = (uintptr_t)a, pb = (uintptr_t)b;
    return a && b && pa < pb + nb && pb < pa + na;
}

/* Whether array k of `arrays` (equal sizes) shares storage with another one. */
inline bool overlaps_another(const void *const *ptr, int arrays, int k, size_t bytes) {
    for (int m = 0; m < arrays; ++m)
        if (m != k && overlap(ptr[k], bytes, ptr[m], bytes)) return true;
    return false;
}

/* Populate the pages of [p, p + bytes) for writing, contents kept: MADV_POPULATE_WRITE, or an atomic
 * OR of 0 into every page where the kernel has no such advice. */
inline void populate_range(char *p, size_t bytes) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    char *a = (char *)((uintptr_t)p & ~(uintptr_t)(page - 1)), *end = p + bytes;
#ifdef MADV_POPULATE_WRITE
    if (madvise(a, (size_t)(end - a), MADV_POPULATE_WRITE) == 0) return;
#endif
    for (; a < end; a += page) __atomic_fetch_or(a < p ? p : a, 0, __ATOMIC_RELAXED);
}

/* The same for the arrays of a call (equal sizes), with threads when there is much of it (zeroing new
 * pages is what takes the time: 104 MB in 9 arrays). */
inline void populate(void *const *ptr, int arrays, size_t bytes) {
    if (bytes == 0 || arrays == 0) return;
    const size_t total = bytes * (size_t)arrays;
    const int nt = (int)std::min<size_t>(8, total / kPopulateChunk);
    auto part = [=](int t, int T) {
        for (int k = 0; k < arrays; ++k) {
            const size_t a = bytes * (size_t)t / T, b = bytes * (size_t)(t + 1) / T;
            if (ptr[k] && b > a) populate_range((char *)ptr[k] + a, b - a);
        }
    };
    int started = 0;
    std::thread th[8];
    try {
        for (; started < nt - 1; ++started) th[started] = std::thread(part, started, nt);
    } catch (...) {     /* no thread to be had: this one does the rest */
    }
    for (int t = started; t < std::max(1, nt); ++t) part(t, std::max(1, nt));
    for (int t = 0; t < started; ++t) th[t].join();
}

struct Arrays {
    int count = 0;
    const uint32_t *src[kMaxArrays];
    uint32_t *dst[kMaxArrays];
};

/* n 4-byte elements of every array: a thread's loads, one per array, are all in flight together. */
static __global__ void k_copy_arrays(int n, Arrays a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t v[kMaxArrays];
#pragma unroll
    for (int k = 0; k < kMaxArrays; ++k)
        if (k < a.count) v[k] = a.src[k][i];
#pragma unroll
    for (int k = 0; k < kMaxArrays; ++k)
        if (k < a.count) a.dst[k][i] = v[k];
}

/* Enqueue the copies of n 4-byte elements src[k] -> dst[k] (null entries are skipped) between host and
 * device: one kernel for the arrays the device can use in place, cudaMemcpyAsync for the others, and for
 * host arrays that share storage (written one after the other, so that the later one's values stay).  The
 * caller synchronises the stream before it returns.  An injected failure of cudaMemcpyAsync (fault_hit)
 * is one of this too, whichever way the arrays go. */
inline mdrl_status copy_arrays(mdrl_ctx *c, int n, int arrays, const void *const *src, void *const *dst, bool to_host) {
    if (fault_hit("cudaMemcpyAsync")) {
        set_error("cudaMemcpyAsync of the call's arrays: injected failure (MDRL_FAULT)");
        return MDRL_ERR_CUDA;
    }
    Arrays a;
    void *fresh[kMaxArrays];
    int nfresh = 0;
    for (int k = 0; k < arrays && n > 0; ++k) {
        if (!src[k] || !dst[k]) continue;
        bool pageable = false;
        void *v = to_host && overlaps_another(dst, arrays, k, 4 * (size_t)n)
                      ? nullptr : device_view(c, to_host ? dst[k] : src[k], 4, &pageable);
        if (!v) {
            MDRL_CUDA(cudaMemcpyAsync(dst[k], src[k], 4 * (size_t)n, to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice,
                                      c->stream));
            continue;
        }
        a.src[a.count] = (const uint32_t *)(to_host ? src[k] : v);
        a.dst[a.count++] = (uint32_t *)(to_host ? v : dst[k]);
        if (pageable && to_host) fresh[nfresh++] = dst[k];
    }
    populate(fresh, nfresh, 4 * (size_t)n);
    if (a.count) k_copy_arrays<<<nblk(n, 256), 256, 0, c->stream>>>(n, a);
    MDRL_CUDA(cudaGetLastError());
    return MDRL_OK;
}

}  // namespace mdrl
