/*
 * mdrl_ctx.cuh — the context structure and host helpers shared by mdrl.cu (single system) and
 * mdrl_batch.cu (batched replicas).
 */
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "mdrl_internal.h"
#include "mdrl_force_list.cuh"

using mdrl::set_error;

namespace mdrl {
struct PmeState;
struct BondedState;
}

#define MDRL_CUDA(call)                                                                   \
    do {                                                                                  \
        if (mdrl::fault_hit(#call)) {                                                     \
            set_error(std::string(#call) + ": injected failure (MDRL_FAULT)");           \
            return MDRL_ERR_CUDA;                                                         \
        }                                                                                 \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));                \
            return MDRL_ERR_CUDA;                                                         \
        }                                                                                 \
    } while (0)

#define MDRL_TRY(expr)                         \
    do {                                       \
        mdrl_status s_ = (expr);               \
        if (s_ != MDRL_OK) return s_;          \
    } while (0)

template <class T>
inline mdrl_status dalloc(T **p, size_t count) {
    if (*p) { cudaFree(*p); *p = nullptr; }
    if (count == 0) return MDRL_OK;
    MDRL_CUDA(cudaMalloc((void **)p, sizeof(T) * count));
    return MDRL_OK;
}

template <class T>
inline void dfree(T **p) {
    if (*p) { cudaFree(*p); *p = nullptr; }
}

struct mdrl_ctx {
    typedef mdrl::Geom Geom;
    typedef mdrl::MassTab MassTab;
    typedef mdrl::UnitOut UnitOut;
    typedef mdrl::DevTotals DevTotals;
    mdrl_params p;
    Geom g;
    int ncells = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t evf0 = nullptr, evf1 = nullptr; /* around the force kernel */

    /* tables */
    int order = 1, nseg = 0, bins = 256, min_log2 = -2;
    bool raw = false;
    bool local = false;          /* coefficients in u = r2 - bin start (MDRL_TABLE_BIN_LOCAL) */
    std::vector<float> tab;      /* canonical [6][order+1][nseg*bins] */
    std::vector<float> pcoef;    /* [T*T*4] */
    float ke = 0.0f;
    float2 *d_f2 = nullptr, *d_e2 = nullptr;
    float4 *d_f4 = nullptr, *d_e4 = nullptr;
    float4 *d_wa = nullptr, *d_wb = nullptr;   /* the one-warp-per-item and list kernels' tables */
    float2 *d_wc = nullptr;
    float *d_w1 = nullptr;
    float4 *d_fr = nullptr;      /* order 1: force functions packed per index (32 B) */
    float4 *d_pcoef = nullptr;
    MassTab mt_half, mt_full;
    MassTab *d_mt = nullptr;     /* device copies: [0] half kick, [1] full kick */

    /* particle buffers */
    int cap = 0, n = 0;
    float *d_ux = nullptr, *d_uy = nullptr, *d_uz = nullptr, *d_uq = nullptr;
    int *d_ut = nullptr;
    int *d_inv = nullptr;   /* cell-order position of each user index (force evaluations) */
    float *d_ox = nullptr, *d_oy = nullptr, *d_oz = nullptr; /* user-order outputs */
    float *d_ovx = nullptr, *d_ovy = nullptr, *d_ovz = nullptr;
    int *d_ocnt = nullptr;
    float4 *d_pos[2] = {nullptr, nullptr}, *d_vel[2] = {nullptr, nullptr};
    int *d_type[2] = {nullptr, nullptr}, *d_id[2] = {nullptr, nullptr};
    int cur = 0;
    int *d_cell_of = nullptr, *d_slot = nullptr, *d_tmp = nullptr, *d_sorted = nullptr;
    int *d_count = nullptr, *d_start = nullptr;
    int *d_work = nullptr;      /* the persistent force kernels' item counters [2], then the list kernel's items [2] */
    int2 *d_tstart = nullptr, *d_tile[2] = {nullptr, nullptr};   /* the list kernel's tiles (Tiles) */
    float *d_narrow = nullptr;  /* the narrow kernel's accumulators for crowded cells */
    bool narrow = false;        /* the state's steps take the narrow kernel (plan_narrow) */
    unsigned *d_key = nullptr;   /* in-cell sort key (Morton code inside the cell) */
    unsigned long long *d_sortkey = nullptr;   /* sorted chunks of cells above kSortSmall */
    unsigned long long *d_F64 = nullptr;
    float *d_F32 = nullptr;
    unsigned long long *d_Fscr64 = nullptr; /* scratch accumulators for mdrl_time_force */
    float *d_Fscr32 = nullptr;
    int *d_cnt = nullptr;
    UnitOut *d_unit = nullptr;
    size_t unit_cap = 0;
    double *d_kepart = nullptr;
    int kecap = 0;
    DevTotals *d_tot = nullptr;
    mdrl::TotScratch *d_totscr = nullptr;   /* k_totals' partial sums */
    DevTotals *h_tot = nullptr;  /* pinned host copies, read back with the results of a call */
    unsigned *h_err = nullptr;
    DevTotals *h_tot_dev = nullptr;  /* the same two, as device addresses */
    unsigned *h_err_dev = nullptr;
    unsigned *d_err = nullptr;
    int num_sms = 0;
    int host_tables = 0;         /* the device walks the host's page tables: pageable memory in place */

    /* pair-eval staging */
    int pcap = 0;
    float4 *d_pr = nullptr, *d_pn = nullptr, *d_pout = nullptr;
    int *d_ptr = nullptr, *d_ptn = nullptr;
    float2 *d_paux = nullptr;

    /* state */
    bool have_state = false;
    /* [k]: one step from buffer slot k to 1-k; [2 + k]: two steps from slot k back to it */
    cudaGraph_t graph[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaGraphExec_t graph_exec[4] = {nullptr, nullptr, nullptr, nullptr};
    int graph_n = -1;
    bool graph_extra = false;

    /* long-range electrostatics (mdrl_set_pme), null when off */
    mdrl::PmeState *pme = nullptr;
    mdrl::BondedState *bonded = nullptr;   /* bonded terms (mdrl_set_bonded), or none */

    /* force-kernel tile (mdrl_set_tile / mdrl_autotune) */
    mdrl_tile tile = {mdrl::kFW, mdrl::kStepsPerPiece, 0};
    bool tile_asked = false;     /* by a caller (the tuner's choice is for dynamics alone) */
    bool batch = false;          /* the buffers of an mdrl_batch (which sizes d_unit itself) */
};

namespace mdrl {
mdrl_status ensure_capacity(mdrl_ctx *c, int n);
TableDev table_dev(const mdrl_ctx *c);
int eff_order(const mdrl_ctx *c);
mdrl_status check_device_errors(mdrl_ctx *c);

/* Raise the dynamic shared-memory limit of a force kernel once per kernel and device. */
mdrl_status prepare_force_kernel(force_fn fn, int device);
/* Whether force evaluations run the list kernel, and its persistent grid: the CTAs that fit on the GPU
 * at once, or fewer when there are fewer items. */
bool list_eval(const mdrl_ctx *c);
/* The totals of the last force launch (its result slots, at most `upto`; nke kinetic-energy partials) into
 * d_tot. */
void launch_totals(mdrl_ctx *c, const TotUnits &units, long long upto, int nke, bool energy);
mdrl_status list_grid(list_fn fn, size_t smem, long long items, bool fine, int num_sms, int *grid);

cudaStream_t pme_stream(const mdrl_ctx *c);    /* PME's own stream, or null without PME */

/* A call that hands the caller's arrays to kernels or copies: on every return before done() it waits for
 * the call's streams, so that the caller may free or reuse the arrays whatever the status.  (Direct
 * calls: an injected failure does not reach them.) */
struct CallGuard {
    mdrl_ctx *c;
    cudaStream_t side;
    bool open = true;
    explicit CallGuard(mdrl_ctx *ctx, cudaStream_t side_stream = nullptr) : c(ctx), side(side_stream) {}
    CallGuard(const CallGuard &) = delete;
    void done() { open = false; }              /* the streams have been joined and waited for */
    ~CallGuard() {
        if (!open) return;
        if (side) (void)cudaStreamSynchronize(side);
        if (cudaStream_t s = pme_stream(c)) (void)cudaStreamSynchronize(s);
        if (c->stream) (void)cudaStreamSynchronize(c->stream);
    }
};
/* 1 while a stream of the context (or `side`) holds work that has not finished. */
int streams_pending(const mdrl_ctx *c, cudaStream_t side = nullptr);
/* PME (mdrl_pme.cu): setup, teardown, the reciprocal part of a force evaluation, its energies. */
mdrl_status pme_setup(mdrl_ctx *c, const mdrl_pme_params *p);
void pme_free(mdrl_ctx *c);
mdrl_status pme_begin(mdrl_ctx *c, int n, const float4 *pos, bool energy);    /* before the pair kernel's launch */
mdrl_status pme_finish(mdrl_ctx *c, int n, const float4 *pos, unsigned long long *F64, float *F32);   /* after it */
mdrl_status pme_add_energy(mdrl_ctx *c, int n);
/* Bonded terms (mdrl_bonded.cu): forces into the accumulators of cell-order buffer pos / pid
 * (after the pair kernel), energies into the totals (after k_totals). */
mdrl_status bonded_enqueue(mdrl_ctx *c, int n, const float4 *pos, const int *pid, unsigned long long *F64,
                           float *F32, bool energy);
mdrl_status bonded_add_energy(mdrl_ctx *c, int n);
mdrl_status bonded_check_atoms(const mdrl_ctx *c, int n);
void bonded_free(mdrl_ctx *c);
mdrl_status upload_tables(mdrl_ctx *c);
/* Tiles: change (re-capturing graphs), and the autotuner's process-wide cache. */
/* allow8: 8-warp CTAs and pruning (fixed point, one system); allow_warp: one warp per item
 * (fixed point) */
mdrl_status set_tile(mdrl_ctx *c, const mdrl_tile *t, bool allow8, bool allow_warp, bool asked);
bool tune_lookup(const std::string &key, mdrl_tile *t);
void tune_store(const std::string &key, const mdrl_tile &t, float ms);
std::string tune_key_common(const mdrl_ctx *c);
}  // namespace mdrl
