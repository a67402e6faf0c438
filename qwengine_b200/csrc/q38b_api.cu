// q38b_api.cu -- host side of libq38b200.so: context, launch planning, C ABI (include/q38b200.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "../../include/q38b200.h"
#include "q38b_act.cuh"
#include "q38b_internal.h"
#include "q38b_topk.cuh"
#include "q38b_gemv1.cuh"

using namespace q38b;

const uint32_t* q38b_grid_source(const q38b_ctx* ctx, uint32_t type) {
    switch (type) {
        case T_IQ3_XXS: return ctx->d_cb_iq3xxs;
        case T_IQ3_S: return ctx->d_cb_iq3s;
        case T_IQ2_XXS: return ctx->d_code16[0];
        case T_IQ2_XS: return ctx->d_code16[1];
        case T_IQ2_S: return ctx->d_code16[2];
        case T_IQ1_S: case T_IQ1_M: return ctx->d_code16[3];
        default: return nullptr;
    }
}

#define Q38B_CUDA(ctx, call)                                   \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess) {                               \
            (ctx)->last_cuda = (int)e_;                        \
            return Q38B_ERR_CUDA;                              \
        }                                                      \
    } while (0)

// Opt-in shared-memory size of a kernel, set once per context (= per device) and kernel; the record lives in the
// context, so two contexts on two devices never disturb each other.
int q38b_ensure_kernel_smem(q38b_ctx* ctx, const void* kern, int dyn_smem_bytes, bool max_carveout) {
    for (int i = 0; i < ctx->n_configured; i++)
        if (ctx->configured[i] == kern) return Q38B_OK;
    Q38B_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_smem_bytes));
    if (max_carveout) Q38B_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    if (ctx->n_configured < (int)(sizeof(ctx->configured) / sizeof(ctx->configured[0]))) ctx->configured[ctx->n_configured++] = kern;
    return Q38B_OK;
}

namespace {

constexpr long long GEMV_PART_ITEMS = 131072;   // (tile, K-part) sums the scratch area of the several-column kernel holds: 64 MB

int align_up(int v, int a) { return (v + a - 1) / a * a; }

bool known_format(uint32_t t) {
    switch (t) {
        case T_Q8_0: case T_Q4_K: case T_Q5_K: case T_Q6_K: case T_IQ3_XXS: case T_IQ3_S: case T_IQ4_XS: return true;
        case T_Q2_K: case T_IQ2_XXS: case T_IQ2_XS: case T_IQ2_S: case T_IQ1_S: case T_IQ1_M: return true;   // one-column kernel, dequantizer, prefill
        default: return false;
    }
}

// alignment (bytes) the shared-memory loads of a format need from W and row_bytes
int format_alignment(uint32_t t) {
    switch (t) {
        case T_Q4_K: case T_Q5_K: return 16;
        case T_IQ4_XS: return 8;
        case T_Q2_K: return 4;
        default: return 2;
    }
}

constexpr int G1_WARPS = 8;                  // consumer warps of a CTA when two CTAs share an SM
// ... when a CTA has the SM to itself (measured on B200: the row-group decoder wants its 80 registers, which 20 warps
// leave it; the others gain from more warps in flight, 5120 x 17408 IQ4_XS 15.7 -> 12.5 us)
constexpr int G1_WARPS_ONE = 24, G1_WARPS_ONE_RG = 20;
// several columns: the columns' activations and sums take registers (Q4_K / Q5_K: 20 a column).  Two columns leave room for 19 warps
// of 96 registers (17408 x 5120 Q5_K, per-32: 25.5 us with the 11 of the wide kernel, 19.3); three and four want 128 (168): 15 (11) warps
constexpr int G1_COLS = 4;
constexpr int g1_warps_cols(int fmt, int sum_cols) { return sum_cols == 2 ? 19 : fmt == T_Q4_K || fmt == T_Q5_K ? 11 : 15; }
constexpr int G1_SMEM_BUDGET = 113 * 1024;   // two CTAs per SM (228 KB of shared memory per SM, 1 KB reserved per CTA)


struct Plan1 {
    Gemv1Args a;
    int grid;
    int smem;
    int rows;   // rows per tile: 8, 4 or 2
    int rg;     // 1: row-group mapping (tables in static shared memory, activations staged twice)
    int occ;    // CTAs per SM: 2 (8 consumer warps) or 1 (24 consumer warps, the whole shared memory)
    int nc;     // columns of the launch
    int sum_cols;   // columns the kernel is built for: 1, 2 or G1_COLS
    int xt;     // 1: expanded grid tables (IQ2 / IQ1)
};

// The row-group decoders want every row to start 8 bytes aligned: W is 16-byte aligned, so the row stride decides.
bool rowgroup_eligible(uint32_t type, size_t row_bytes, int rows) { return type == T_IQ3_XXS && row_bytes % 8 == 0 && rows % 4 == 0; }

// Shared-memory carve-up of the single-column kernel: barriers | activation scales | activations | codebook |
// per-tile slice sums | ring of stages (8 row slots of one 1024-weight slice each).
int plan_gemv1_rows(const q38b_ctx* ctx, uint32_t type, int K, const int* Ms, int n_mats, size_t row_bytes, int G1_ROWS, int occ, int nc, int xt, Plan1* p, int sum_cols = 1) {
    const int bb = block_bytes((int)type);
    p->occ = occ;
    p->xt = xt;
    p->nc = nc;
    p->a.nc = nc;
    p->sum_cols = sum_cols;
    const int nsb = K / 256;
    const int rg = nc == 1 && ctx->rowgroup && rowgroup_eligible(type, row_bytes, G1_ROWS) ? 1 : 0;
    const int warps = nc > 1 ? g1_warps_cols((int)type, sum_cols) : occ == 1 ? (rg ? G1_WARPS_ONE_RG : G1_WARPS_ONE) : G1_WARPS;
    const int cb_entries = rg ? 0 : type == T_IQ3_XXS ? 256 : type == T_IQ3_S ? 512 : 0;   // row groups keep their tables in static shared memory
    const int budget = (occ == 1 ? ctx->smem_optin : std::min(ctx->smem_optin, G1_SMEM_BUDGET)) - 128 - (rg ? RG_STATIC_BYTES : 0);
    Gemv1Args& a = p->a;
    p->rows = G1_ROWS;
    p->rg = rg;
    a.nsb = nsb;
    a.n_slices = (nsb + 3) / 4;
    a.n_tiles = 0;
    for (int i = 0; i < G1_MAX_MATS; i++) {
        a.tile_start[i] = a.n_tiles;
        if (i < n_mats) a.n_tiles += (Ms[i] + G1_ROWS - 1) / G1_ROWS;
    }
    for (int i = n_mats; i < G1_MAX_MATS; i++) a.tile_start[i] = a.n_tiles;
    a.off_actd = 1664;   // barriers (1536 bytes), flags
    a.off_actq = a.off_actd + nc * a.n_slices * 4 * 32;
    a.off_cb = a.off_actq + nc * a.n_slices * (rg ? 4 * ACTR_BLOCK_BYTES : 1024);
    const int packed = nsb * bb;
    // stage shape: 8 whole rows in one bulk copy when the rows are packed and small enough, else 8 per-row copies of a
    // K-chunk of `chunk_slices` slices (bulk copies are issue-rate limited: keep each above ~2 KB)
    const int target = occ == 1 ? 40 * 1024 : 28 * 1024;
    if ((long long)row_bytes == packed && G1_ROWS * packed <= target) {
        a.contiguous = 1;
        a.chunk_slices = a.n_slices;
        a.slot_stride = packed;
        a.stage_bytes = align_up(G1_ROWS * packed + 64, 128);
    } else {
        a.contiguous = 0;
        int cs = std::max(1, std::min(a.n_slices, (target / G1_ROWS - 32) / (4 * bb)));
        const int nch = (a.n_slices + cs - 1) / cs;
        cs = (a.n_slices + nch - 1) / nch;          // even chunks
        a.chunk_slices = cs;
        a.slot_stride = align_up(cs * 4 * bb + 32, 16);
        a.stage_bytes = align_up(G1_ROWS * a.slot_stride + 64, 128);
    }
    a.n_chunks = (a.n_slices + a.chunk_slices - 1) / a.chunk_slices;
    const int min_stages = (warps + a.chunk_slices - 1) / a.chunk_slices + 1;
    for (int rep_log2 = cb_entries ? cb1_rep_log2((int)type) : 0; rep_log2 >= (cb_entries ? cb1_rep_log2((int)type) : 0); rep_log2--) {   // the replica count is part of the format's decoder
        a.cb_rep_log2 = rep_log2;
        a.off_sgn = a.off_cb + align_up((cb_entries * 4 << rep_log2) + (xt ? gridx_bytes((int)type) : 2 * code16_entries((int)type)), 128);
        a.off_red = a.off_sgn + ((type == T_IQ3_XXS && !rg) || (xt && gridx_signs((int)type)) ? KSIGN_TABLE_BYTES : 0);
        for (int stages = G1_MAX_STAGES; stages >= min_stages; stages--) {
            // tile buffers: a warp can run at most (stages + warps) units ahead of a tile that is still being finished
            const int tb = (warps + stages * a.chunk_slices + 2 * a.n_slices - 1) / a.n_slices + 1;
            if (tb > G1_MAX_TILEBUF) continue;
            a.off_stage = align_up(a.off_red + tb * a.n_slices * G1_ROWS * sum_cols * 4, 128);
            if (a.off_stage + stages * a.stage_bytes + align_up(3 * bb, 128) > budget) continue;
            a.n_stages = stages;
            a.n_tilebuf = tb;
            p->smem = a.off_stage + stages * a.stage_bytes + 128 + align_up(3 * bb, 128);   // granules past a ragged row end are read (and discarded)
            p->grid = std::max(1, std::min(occ * ctx->sm_count, a.n_tiles));
            return Q38B_OK;
        }
        if (!cb_entries) break;
    }
    return Q38B_ERR_NOMEM;
}

// Whether the expanded grids pay: they are 64 KB a CTA to fill before its first row.  The IQ2 formats gain from the
// smallest matrices on; IQ1 has less to gain: IQ1_M takes them from seven of a tile's slices per SM on (2048 x 1024 6.1 us with
// the codes, 6.5 with the grids; 4096 x 2048 6.7 us either way; 6144 x 8192 14.7 and 13.0 us), IQ1_S from four tiles a CTA on
// (2048 x 1024 5.9 and 6.2 us, 4096 x 4096 7.0 and 7.3 us, 6144 x 4096 8.8 and 8.4 us).
bool gridx_pays(const q38b_ctx* ctx, uint32_t type, int K, const int* Ms, int n_mats) {
    if (type != T_IQ1_S && type != T_IQ1_M) return gridx_copies((int)type) > 0;
    long long tiles = 0;
    for (int i = 0; i < n_mats; i++) tiles += (Ms[i] + 7) / 8;
    return type == T_IQ1_S ? tiles >= 4 * ctx->sm_count : tiles * ((K + 1023) / 1024) >= 7 * ctx->sm_count;
}

// Rows per tile: the largest of 8, 4, 2 that can be planned.  Measured on B200 for every shape of the benchmark pass,
// eight rows win even where fewer rows would balance the CTAs better or let a tile be fetched by one copy: the cost per
// (tile, slice) unit (activation loads, waits, lane reduction) outweighs both.
// One CTA per SM with three times the consumer warps (ctx->one_cta, on by default) is tried first: one set of tables and
// one quantized column per SM, deeper rings, 16-row tiles for the row groups.  Measured on B200 it is faster than two
// CTAs per SM for every shape of the benchmark pass (4.23 ms against 4.30 ms with only long rows and row groups on it,
// 5.2 ms with none); the two-CTA plans remain for shapes whose one-CTA plan does not fit.
// The expanded grids of IQ2 / IQ1 (64 KB, for two formats 16 KB of sign masks) are taken where tiles of eight, four or two
// rows fit beside them (5120 x 45056 IQ2_XS: 39.6 us in tiles of four, 61.3 us with the codes in tiles of eight); longer rows
// (from 63,744 weights on) keep the 16-bit codes and with them every length that has a plan.
int plan_gemv1(const q38b_ctx* ctx, uint32_t type, int K, const int* Ms, int n_mats, size_t row_bytes, Plan1* best) {
    if (ctx->one_cta) {
        const int cands1[4] = {16, 8, 4, 2};
        for (int xt = gridx_pays(ctx, type, K, Ms, n_mats); xt >= 0; xt--) {
            for (int rows : cands1) {
                if (rows == 16 && !(ctx->rowgroup && rowgroup_eligible(type, row_bytes, 16))) continue;
                memset(best, 0, sizeof(*best));
                if (plan_gemv1_rows(ctx, type, K, Ms, n_mats, row_bytes, rows, 1, 1, xt, best) == Q38B_OK) return Q38B_OK;
            }
        }
    }
    const int cands[3] = {8, 4, 2};
    for (int rows : cands) {
        memset(best, 0, sizeof(*best));
        if (plan_gemv1_rows(ctx, type, K, Ms, n_mats, row_bytes, rows, 2, 1, 0, best) == Q38B_OK) return Q38B_OK;
    }
    return Q38B_ERR_NOMEM;
}

// what cols_by_granule can ask for with Q8_K blocks; per-32 columns: every format
constexpr bool granule_cols_q8k(int fmt, int sum_cols) {
    return one_column_only(fmt) || fmt == T_Q8_0 || (sum_cols == 2 && (fmt == T_Q5_K || fmt == T_Q6_K));
}
// Two to four columns in one launch: one CTA per SM, tiles of eight rows.  Two columns that the kernel for two has no room for (its
// 19 warps want a longer ring) take the one for four.
int plan_gemv1_cols(const q38b_ctx* ctx, uint32_t type, int K, const int* Ms, int n_mats, size_t row_bytes, int nc, bool a32, Plan1* p) {
    if (!ctx->one_cta) return Q38B_ERR_NOMEM;
    for (int sum_cols = nc == 2 ? 2 : G1_COLS; sum_cols <= G1_COLS; sum_cols += 2) {
        if (!a32 && !granule_cols_q8k((int)type, sum_cols)) continue;
        memset(p, 0, sizeof(*p));
        if (plan_gemv1_rows(ctx, type, K, Ms, n_mats, row_bytes, 8, 1, nc, gridx_copies((int)type) > 0, p, sum_cols) == Q38B_OK) return Q38B_OK;
    }
    return Q38B_ERR_NOMEM;
}

// Whether n = 2..4 columns on `rows` rows of nsb super-blocks take this kernel, which decodes a granule once for all of them and pays
// a dp4a for each, instead of the several-column kernel, whose fragments cost the same for one column as for eight.  Same bits
// either way; rows in K-parts never (other sums).  The lines are where the two met over 1024 to 65536 rows of 1024 to 17408 weights:
// more warps and tables make this kernel's start longer (1024 x 1024: 5.0 to 6.5 us against 3.9 to 4.3), tiles of eight rows feed
// more SMs where rows are few and long (1024 x 8192 IQ2_S: 1.26 times as fast).  Two columns of Q8_K blocks (several-column kernel
// first, us): 17408 x 5120 IQ1_M 27.1 / 21.0, IQ2_S 24.8 / 22.0, Q5_K 20.2 / 18.6, Q6_K 26.3 / 21.1, but Q4_K 15.1 / 16.1 and 17408 x 2816
// IQ2_XXS 14.6 / 15.0; Q2_K 5120 x 8192 12.4 / 13.2, x 17408 24.1 / 21.4.  Per-32 columns, which the other kernel scales every 32 weights
// in floats: 17408 x 5120 Q2_K 24.9 / 17.8, Q4_K 20.2 / 16.4, IQ3_XXS 25.4 / 23.0, but IQ3_S 26.8 / 27.0 and 17408 x 1024 Q4_K 8.5 / 10.9.
// Three and four columns gain less: Q8_0, whose fragments are scaled every 32 weights (5120 x 8192, three 18.2 / 15.8, four 18.5 / 17.2),
// and long rows, whose activations leave the other kernel a short ring (5120 x 17408, per-32, three columns Q2_K 33.7 / 28.9, IQ1_M
// 36.3 / 32.5; four IQ2_S 39.9 / 37.5).
bool cols_by_granule(const q38b_ctx* ctx, uint32_t type, long long rows, int nsb, int n, bool a32) {
    constexpr int NEVER = 1 << 30;
    if ((!a32 && q38b_cols_in_parts(type, 256 * nsb)) || ctx->cols_route == 1) return false;
    if (ctx->cols_route == 2) return true;
    const bool few = rows <= 2048, many = rows >= 8192;
    int from = NEVER;   // the shortest row
    if (n == 2) {
        switch (type) {
            case T_Q8_0: from = many ? 4 : 8; break;
            case T_Q6_K: from = few ? 11 : 8; break;
            case T_IQ1_M: case T_IQ2_S: case T_IQ2_XS: from = few ? 20 : 8; break;
            case T_IQ1_S: from = !few ? 16 : a32 ? 20 : 32; break;
            case T_IQ2_XXS: from = a32 ? (few ? 20 : 16) : few ? 32 : 40; break;
            case T_Q2_K: from = a32 ? (few ? 20 : 8) : few ? 32 : 49; break;
            case T_Q4_K: from = a32 ? (few ? 11 : 8) : NEVER; break;
            case T_Q5_K: from = a32 ? (few ? 11 : 8) : few ? 32 : many ? 20 : NEVER; break;
            case T_IQ3_XXS: from = !a32 ? NEVER : few ? 32 : many ? 16 : 40; break;
            case T_IQ4_XS: from = !a32 ? NEVER : few ? 20 : many ? 8 : 40; break;
            default: from = !a32 ? NEVER : few ? 32 : 40; break;   // IQ3_S
        }
    } else {
        switch (type) {
            case T_Q8_0: from = n == 4 ? 24 : rows >= 16384 ? 4 : 20; break;
            case T_Q2_K: from = a32 ? (n == 3 ? 20 : 64) : NEVER; break;
            case T_IQ1_M: from = n == 3 ? 32 : 64; break;
            case T_IQ2_S: from = n == 3 ? 48 : a32 ? 64 : NEVER; break;
            case T_IQ2_XS: from = n == 3 ? 48 : NEVER; break;
            default: break;
        }
    }
    return nsb >= from;
}

// Whether one column with per-32 activations takes the plan `p` of one CTA per SM (else two).  These calls follow one another
// without overlap, so a launch's start counts: where a row has few slices, or an SM one tile, two CTAs fill twice as many
// small stages while the tables are set up (17408 x 1024 Q4_K: 7.6 us, one CTA 10.8 us; Q2_K 7.9 and 10.8 us; 1024 x 5120 Q4_K
// 4.0 and 4.4 us); where there is more, the single set of tables and the longer ring win (5120 x 17408 IQ2_XS 29.1 and 18.6
// us, IQ4_XS 21.1 and 16.9 us).  The lines are where the two met over 512 to 17408 rows of 512 to 17408 weights: the
// expanded grids of IQ2 pay earliest; Q5_K and Q6_K lose with chunks of four slices (17408 x 8192 Q5_K: two CTAs 22.2 us, one
// 28.0 us); Q4_K, which has the least to decode, gains on many rows at five and six slices only (17408 x 11008: 23.8 and
// 28.2 us), IQ3_XXS from 14 on.
bool act_q8_one_cta(const q38b_ctx* ctx, uint32_t type, const Plan1& p) {
    const int n = p.a.n_slices, tiles = p.a.n_tiles, sms = ctx->sm_count;
    switch (type) {
        case T_Q8_0: return false;
        case T_IQ2_XXS: case T_IQ2_XS: case T_IQ2_S: return n >= 3 || tiles <= 4 * sms;
        case T_IQ1_M: return n >= 3;
        case T_IQ4_XS: return n >= 4;
        default: break;
    }
    if (tiles <= sms) return n >= 11;
    switch (type) {
        case T_Q5_K: case T_Q6_K: return n >= 3 && p.a.chunk_slices != 4;
        case T_Q4_K: return n == 5 || n == 6 || (n >= 11 && tiles <= 3 * sms);
        case T_IQ3_XXS: return n >= 14;
        default: return n >= 5;   // IQ1_S, IQ3_S, Q2_K
    }
}

// How many of `left` columns the next launch of this kernel takes (Q6_K with per-32 activations, which has no other), with its plan
// in *p when that is more than one: the most that fit shared memory, at most four; six are two threes.
int next_cols(const q38b_ctx* ctx, uint32_t type, int K, int M, size_t row_bytes, int left, Plan1* p) {
    int n = left == 6 ? 3 : std::min(G1_COLS, left);
    while (n > 1 && plan_gemv1_cols(ctx, type, K, &M, 1, row_bytes, n, true, p) != Q38B_OK) n--;
    return n;
}

// The next launch of `left` columns that keep the one-column kernel's bits: how many it takes (1: that kernel's single column) and
// whether they go to the kernel that decodes a granule for all of them (its plan in *p).
int next_launch(const q38b_ctx* ctx, uint32_t type, int K, const int* M, int n_mats, size_t row_bytes, int left, bool a32, bool* granule, Plan1* p) {
    long long rows = 0;
    for (int i = 0; i < n_mats; i++) rows += M[i];
    auto by_granule = [&](int n) {
        return n >= 2 && n <= G1_COLS && cols_by_granule(ctx, type, rows, K / 256, n, a32) && plan_gemv1_cols(ctx, type, K, M, n_mats, row_bytes, n, a32, p) == Q38B_OK;
    };
    *granule = by_granule(left);
    if (*granule || left == 1) return left;
    if (a32 && type == T_Q6_K) {
        const int n = next_cols(ctx, type, K, M[0], row_bytes, left, p);
        *granule = n > 1;
        return n;
    }
    const int n = std::max(1, q38b_cols_take(ctx, type, K, M, n_mats, row_bytes, left, a32));
    *granule = n < left && by_granule(n);
    return n;
}

template <int FMT, int ROWS, bool RG, bool A32 = false, int OCC = 2, int NC = 1, bool XT = false>
int launch_gemv1_rows(q38b_ctx* ctx, const Plan1& p, cudaStream_t st) {
    constexpr int WARPS = NC > 1 ? g1_warps_cols(FMT, NC) : OCC == 1 ? (RG ? G1_WARPS_ONE_RG : G1_WARPS_ONE) : G1_WARPS;
    auto kern = gemv1_kernel<FMT, WARPS, ROWS, RG, A32, OCC, NC, XT>;
    const int rc = q38b_ensure_kernel_smem(ctx, (const void*)kern, (OCC == 1 ? ctx->smem_optin : G1_SMEM_BUDGET) - (RG ? RG_STATIC_BYTES : 0), true);
    if (rc != Q38B_OK) return rc;
    if (ctx->check_occupancy) {   // test hook: count launches whose CTAs would not be resident as often as planned
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * (1 + WARPS), (size_t)p.smem) != cudaSuccess || per_sm < OCC)
            ctx->occupancy_shortfalls++;
    }
    const Gemv1Args& args = p.a;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3(32 * (1 + WARPS));
    cfg.dynamicSmemBytes = (size_t)p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl ? 1 : 0;
    Q38B_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, args));
    return Q38B_OK;
}

template <int FMT>
int launch_gemv1(q38b_ctx* ctx, const Plan1& p, cudaStream_t st) {
    constexpr bool X = gridx_copies(FMT) > 0;
    if (p.nc > 1) {
        if (p.a.xd32) return p.sum_cols == 2 ? launch_gemv1_rows<FMT, 8, false, true, 1, 2, X>(ctx, p, st) : launch_gemv1_rows<FMT, 8, false, true, 1, G1_COLS, X>(ctx, p, st);
        if constexpr (granule_cols_q8k(FMT, 2)) {
            if (p.sum_cols == 2) return launch_gemv1_rows<FMT, 8, false, false, 1, 2, X>(ctx, p, st);
        }
        if constexpr (granule_cols_q8k(FMT, G1_COLS)) return launch_gemv1_rows<FMT, 8, false, false, 1, G1_COLS, X>(ctx, p, st);
        return Q38B_ERR_ARG;
    }
    if (p.a.xd32) {   // per-32 activations: lane-per-granule mapping only
        if (p.rg) return Q38B_ERR_ARG;
        if constexpr (FMT != T_Q8_0) {
            if (p.occ == 1) return p.rows == 8 ? launch_gemv1_rows<FMT, 8, false, true, 1, 1, X>(ctx, p, st) : Q38B_ERR_ARG;
        }
        if (p.occ == 1) return Q38B_ERR_ARG;
        switch (p.rows) {
            case 8: return launch_gemv1_rows<FMT, 8, false, true>(ctx, p, st);
            case 4: return launch_gemv1_rows<FMT, 4, false, true>(ctx, p, st);
            case 2: return launch_gemv1_rows<FMT, 2, false, true>(ctx, p, st);
            default: return Q38B_ERR_ARG;
        }
    }
    if constexpr (FMT == T_IQ3_XXS) {
        if (p.rg && p.occ == 1 && p.rows == 16) return launch_gemv1_rows<FMT, 16, true, false, 1>(ctx, p, st);
        if (p.rg && p.occ == 1 && p.rows == 8) return launch_gemv1_rows<FMT, 8, true, false, 1>(ctx, p, st);
        if (p.rg && p.occ == 1 && p.rows == 4) return launch_gemv1_rows<FMT, 4, true, false, 1>(ctx, p, st);
        if (p.rg && p.rows == 8) return launch_gemv1_rows<FMT, 8, true>(ctx, p, st);
        if (p.rg && p.rows == 4) return launch_gemv1_rows<FMT, 4, true>(ctx, p, st);
    }
    if (p.occ == 1) {
        if constexpr (X) {
            if (p.xt) {
                switch (p.rows) {
                    case 8: return launch_gemv1_rows<FMT, 8, false, false, 1, 1, true>(ctx, p, st);
                    case 4: return launch_gemv1_rows<FMT, 4, false, false, 1, 1, true>(ctx, p, st);
                    case 2: return launch_gemv1_rows<FMT, 2, false, false, 1, 1, true>(ctx, p, st);
                    default: return Q38B_ERR_ARG;
                }
            }
        }
        switch (p.rows) {
            case 8: return launch_gemv1_rows<FMT, 8, false, false, 1>(ctx, p, st);
            case 4: return launch_gemv1_rows<FMT, 4, false, false, 1>(ctx, p, st);
            case 2: return launch_gemv1_rows<FMT, 2, false, false, 1>(ctx, p, st);
            default: return Q38B_ERR_ARG;
        }
    }
    switch (p.rows) {
        case 8: return launch_gemv1_rows<FMT, 8, false>(ctx, p, st);
        case 4: return launch_gemv1_rows<FMT, 4, false>(ctx, p, st);
        case 2: return launch_gemv1_rows<FMT, 2, false>(ctx, p, st);
        default: return Q38B_ERR_ARG;
    }
}

int dispatch_gemv1(q38b_ctx* ctx, uint32_t type, const Plan1& p1, cudaStream_t st) {
    switch (type) {
        case T_Q8_0: return launch_gemv1<T_Q8_0>(ctx, p1, st);
        case T_Q4_K: return launch_gemv1<T_Q4_K>(ctx, p1, st);
        case T_Q5_K: return launch_gemv1<T_Q5_K>(ctx, p1, st);
        case T_Q6_K: return launch_gemv1<T_Q6_K>(ctx, p1, st);
        case T_IQ3_XXS: return launch_gemv1<T_IQ3_XXS>(ctx, p1, st);
        case T_IQ3_S: return launch_gemv1<T_IQ3_S>(ctx, p1, st);
        case T_IQ4_XS: return launch_gemv1<T_IQ4_XS>(ctx, p1, st);
        case T_Q2_K: return launch_gemv1<T_Q2_K>(ctx, p1, st);
        case T_IQ2_XXS: return launch_gemv1<T_IQ2_XXS>(ctx, p1, st);
        case T_IQ2_XS: return launch_gemv1<T_IQ2_XS>(ctx, p1, st);
        case T_IQ2_S: return launch_gemv1<T_IQ2_S>(ctx, p1, st);
        case T_IQ1_S: return launch_gemv1<T_IQ1_S>(ctx, p1, st);
        case T_IQ1_M: return launch_gemv1<T_IQ1_M>(ctx, p1, st);
        default: return Q38B_ERR_UNSUPPORTED;
    }
}

}  // namespace

extern "C" {

int q38b_ctx_create(int device, q38b_ctx** out) {
    if (!out) return Q38B_ERR_ARG;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0 || device < 0 || device >= n) return Q38B_ERR_NO_DEVICE;
    q38b_ctx* c = new (std::nothrow) q38b_ctx;
    if (!c) return Q38B_ERR_NOMEM;
    c->device = device;
    int rc = Q38B_OK;
    do {
        if (cudaSetDevice(device) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
        cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, device);
        cudaDeviceGetAttribute(&c->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
        if (cudaMalloc(&c->d_status, sizeof(int)) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
        cudaMemset(c->d_status, 0, sizeof(int));
        const void *xxs = nullptr, *s = nullptr;
        if (cudaGetSymbolAddress((void**)&xxs, q38b_iq3xxs_grid) != cudaSuccess ||
            cudaGetSymbolAddress((void**)&s, q38b_iq3s_grid) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
        c->d_cb_iq3xxs = (uint32_t*)xxs;
        c->d_cb_iq3s = (uint32_t*)s;
        const void* t16[4] = {nullptr, nullptr, nullptr, nullptr};
        if (cudaGetSymbolAddress((void**)&t16[0], q38b_iq2xxs_codes) != cudaSuccess || cudaGetSymbolAddress((void**)&t16[1], q38b_iq2xs_codes) != cudaSuccess ||
            cudaGetSymbolAddress((void**)&t16[2], q38b_iq2s_codes) != cudaSuccess || cudaGetSymbolAddress((void**)&t16[3], q38b_iq1s_codes) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
        for (int i = 0; i < 4; i++) c->d_code16[i] = (const uint32_t*)t16[i];
        // candidate lists of q38b_topk: 8 columns x TOPK_MAX_CHUNKS lists x TOPK_MAX_K pairs (1.5 MB), so that the decode path never allocates
        c->part_items = GEMV_PART_ITEMS;
        if (cudaMalloc(&c->d_parts, (size_t)GEMV_PART_ITEMS * 128 * sizeof(float)) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
        if (cudaMemset(c->d_parts, 0xFF, (size_t)GEMV_PART_ITEMS * 128 * sizeof(float)) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }   // PART_EMPTY
        if (cudaMalloc(&c->d_part_count, (size_t)GEMV_PART_ITEMS * sizeof(int)) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
        if (cudaMemset(c->d_part_count, 0, (size_t)GEMV_PART_ITEMS * sizeof(int)) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
        if (cudaMalloc(&c->d_topk, (size_t)8 * TOPK_MAX_CHUNKS * TOPK_MAX_K * sizeof(TopkPair)) != cudaSuccess) { rc = Q38B_ERR_CUDA; break; }
    } while (0);
    if (rc != Q38B_OK) {
        c->last_cuda = (int)cudaGetLastError();
        if (c->d_status) cudaFree(c->d_status);
        if (c->d_topk) cudaFree(c->d_topk);
        if (c->d_parts) cudaFree(c->d_parts);
        if (c->d_part_count) cudaFree(c->d_part_count);
        delete c;
        return rc;
    }
    *out = c;
    return Q38B_OK;
}

void q38b_ctx_destroy(q38b_ctx* ctx) {
    if (!ctx) return;
    if (ctx->d_status) cudaFree(ctx->d_status);
    if (ctx->d_topk) cudaFree(ctx->d_topk);
    if (ctx->d_parts) cudaFree(ctx->d_parts);
    if (ctx->d_part_count) cudaFree(ctx->d_part_count);
    if (ctx->d_flags) cudaFree(ctx->d_flags);
    delete ctx;
}

int q38b_ctx_check(q38b_ctx* ctx, void* stream) {
    if (!ctx) return Q38B_ERR_ARG;
    int bits = 0;
    Q38B_CUDA(ctx, cudaMemcpyAsync(&bits, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    Q38B_CUDA(ctx, cudaStreamSynchronize((cudaStream_t)stream));
    if (bits) {
        Q38B_CUDA(ctx, cudaMemsetAsync(ctx->d_status, 0, sizeof(int), (cudaStream_t)stream));
        // a multi-column matvec that gave up may have left K-part sums and counts behind: back to the resting state
        Q38B_CUDA(ctx, cudaMemsetAsync(ctx->d_parts, 0xFF, (size_t)GEMV_PART_ITEMS * 128 * sizeof(float), (cudaStream_t)stream));
        Q38B_CUDA(ctx, cudaMemsetAsync(ctx->d_part_count, 0, (size_t)GEMV_PART_ITEMS * sizeof(int), (cudaStream_t)stream));
        return Q38B_ERR_DEVICE_WAIT;
    }
    return Q38B_OK;
}

int q38b_last_cuda_error(const q38b_ctx* ctx) { return ctx ? ctx->last_cuda : 0; }

int q38b_ctx_set_static_weights(q38b_ctx* ctx, int enabled) {
    if (!ctx) return Q38B_ERR_ARG;
    ctx->static_weights = enabled ? 1 : 0;
    return Q38B_OK;
}

int q38b_ctx_set_uniform_columns(q38b_ctx* ctx, int enabled) {
    if (!ctx) return Q38B_ERR_ARG;
    ctx->uniform_columns = enabled ? 1 : 0;
    return Q38B_OK;
}

// Test hook (not in the public header): 0 keeps the one-column kernel on its lane-per-granule mapping for every format,
// so that tests and timings can compare the two mappings on the same inputs.
int q38b_debug_set_rowgroup(q38b_ctx* ctx, int enabled) {
    if (!ctx) return Q38B_ERR_ARG;
    ctx->rowgroup = enabled ? 1 : 0;
    return Q38B_OK;
}
// Test hook: one CTA per SM for the one-column kernel: 0 never, otherwise wherever such a plan fits (the default).
int q38b_debug_set_one_cta(q38b_ctx* ctx, int mode) {
    if (!ctx || mode < 0 || mode > 2) return Q38B_ERR_ARG;
    ctx->one_cta = mode ? 1 : 0;
    return Q38B_OK;
}
// Test hook: the multi-column kernel's K-part scratch area counts as `items` (tile, part) sums (0: its real size), so that
// the launch per block of rows that very tall matrices take can be reached with a small one.
int q38b_debug_set_gemv_part_items(q38b_ctx* ctx, long long items) {
    if (!ctx || items < 0 || items > GEMV_PART_ITEMS) return Q38B_ERR_ARG;
    ctx->part_items = items ? items : GEMV_PART_ITEMS;
    return Q38B_OK;
}
// Test hook: enabled = 1 starts counting one-column launches whose CTAs fit an SM less often than their plan assumes;
// returns the count so far.
int q38b_debug_occupancy_shortfalls(q38b_ctx* ctx, int enabled) {
    if (!ctx) return -1;
    ctx->check_occupancy = enabled ? 1 : 0;
    return ctx->occupancy_shortfalls;
}

int q38b_ctx_set_wait_budget_cycles(q38b_ctx* ctx, long long cycles) {
    if (!ctx || cycles < 1000) return Q38B_ERR_ARG;
    ctx->wait_budget_cycles = cycles;
    return Q38B_OK;
}

// Test hook: makes this context believe it is rank 0 of 2 whose peer's flag block is its own arena, which nobody
// signals, so that a cross-GPU barrier runs into its bounded wait on one GPU (enabled = 0 undoes it).
int q38b_debug_fake_silent_peer(q38b_ctx* ctx, int enabled) {
    if (!ctx) return Q38B_ERR_ARG;
    if (enabled) {
        if (!ctx->d_flags) {
            unsigned char handle[64];
            const int rc = q38b_peer_arena_create(ctx, 1 << 20, handle);
            if (rc != Q38B_OK) return rc;
        }
        ctx->peer_flags[0] = ctx->d_flags;
        ctx->peer_flags[1] = ctx->d_flags + 64;   // rank 1 "writes" into words nobody reads; its own word [1] of the local block stays 0
        ctx->n_ranks = 2;
        ctx->rank = 0;
        ctx->peers_connected = 1;
    } else {
        ctx->n_ranks = 1;
        ctx->rank = 0;
        ctx->peers_connected = 0;
    }
    return Q38B_OK;
}

int q38b_ctx_set_pdl(q38b_ctx* ctx, int enabled) {
    if (!ctx) return Q38B_ERR_ARG;
    ctx->pdl = enabled ? 1 : 0;
    ctx->pass_pdl = enabled ? 1 : 0;
    return Q38B_OK;
}

const char* q38b_status_string(int s) {
    switch (s) {
        case Q38B_OK: return "ok";
        case Q38B_ERR_ARG: return "invalid argument";
        case Q38B_ERR_UNSUPPORTED: return "format has no kernel";
        case Q38B_ERR_ALIGN: return "pointer or stride misaligned for the format";
        case Q38B_ERR_CUDA: return "CUDA runtime error";
        case Q38B_ERR_DEVICE_WAIT: return "a bounded device-side wait ran out";
        case Q38B_ERR_NOMEM: return "shape does not fit the shared-memory plan";
        case Q38B_ERR_NO_DEVICE: return "no CUDA device (there is no CPU fallback)";
        default: return "unknown status";
    }
}

int q38b_format_supported(uint32_t type) { return known_format(type) ? 1 : 0; }

size_t q38b_row_bytes(uint32_t type, int K) {
    if (!known_format(type) || K <= 0 || K % 256) return 0;
    return (size_t)(K / 256) * (size_t)block_bytes((int)type);
}

size_t q38b_q8k_bytes(int K) { return K > 0 && K % 256 == 0 ? (size_t)(K / 256) * Q8K_BYTES : 0; }

int q38b_quantize_q8k(q38b_ctx* ctx, const float* x, long long x_ld, int K, int n_rows, void* q8k, long long q8k_stride,
                      void* stream) {
    if (!ctx || !x || !q8k || K <= 0 || K % 256 || n_rows < 1 || x_ld < K || q8k_stride < K / 256) return Q38B_ERR_ARG;
    if (((uintptr_t)x | (uintptr_t)q8k) & 3) return Q38B_ERR_ALIGN;
    const long long blocks = (long long)n_rows * (K / 256);
    quantize_q8k_kernel<<<(unsigned)((blocks + ACT_WARPS - 1) / ACT_WARPS), ACT_WARPS * 32, 0, (cudaStream_t)stream>>>(
        x, x_ld, K, n_rows, (uint8_t*)q8k, q8k_stride);
    Q38B_CUDA(ctx, cudaGetLastError());
    return Q38B_OK;
}

// takes the cross-GPU barrier the planner left for the next launch, if any
static PeerSync take_pending_sync(q38b_ctx* ctx) {
    PeerSync ps;
    memset(&ps, 0, sizeof(ps));
    if (ctx->pending_sync_seq >= 0 && ctx->n_ranks > 1 && ctx->peers_connected) {
        ps.local = ctx->d_flags;
        for (int r = 0; r < 8; r++) ps.peer[r] = ctx->peer_flags[r];
        ps.n = ctx->n_ranks;
        ps.rank = ctx->rank;
        ps.seq = ctx->pending_sync_seq;
        ps.budget = ctx->wait_budget_cycles;
    }
    ctx->pending_sync_seq = -1;
    return ps;
}

int q38b_swiglu_q8k(q38b_ctx* ctx, const float* g, const float* u, long long ld, int n, int n_rows, float* h, void* q8k,
                    long long q8k_stride, void* stream) {
    if (!ctx || !g || !u || n <= 0 || n % 256 || n_rows < 1 || ld < n || (q8k && q8k_stride < n / 256)) return Q38B_ERR_ARG;
    if (((uintptr_t)g | (uintptr_t)u | (uintptr_t)h | (uintptr_t)q8k) & 3) return Q38B_ERR_ALIGN;
    const long long blocks = (long long)n_rows * (n / 256);
    swiglu_q8k_kernel<<<(unsigned)((blocks + ACT_WARPS - 1) / ACT_WARPS), ACT_WARPS * 32, 0, (cudaStream_t)stream>>>(
        g, u, ld, n, n_rows, h, (uint8_t*)q8k, q8k_stride, take_pending_sync(ctx), ctx->d_status);
    Q38B_CUDA(ctx, cudaGetLastError());
    return Q38B_OK;
}

int q38b_add_rmsnorm_q8k(q38b_ctx* ctx, float* x, const float* a, const float* b, const float* w, int n, long long ld, int n_rows, float eps,
                         float* xn, void* q8k, long long q8k_stride, void* stream) {
    if (!ctx || !x || !w || n <= 0 || n % 256 || n > 32 * 256 || ld < n || ld % 4 || n_rows < 1 || (q8k && q8k_stride < n / 256)) return Q38B_ERR_ARG;
    if (((uintptr_t)x | (uintptr_t)a | (uintptr_t)b | (uintptr_t)w | (uintptr_t)xn) & 15) return Q38B_ERR_ALIGN;
    if ((uintptr_t)q8k & 3) return Q38B_ERR_ALIGN;
    add_rmsnorm_q8k_kernel<<<(unsigned)n_rows, (unsigned)(n / 256) * 32, 0, (cudaStream_t)stream>>>(x, a, b, w, n, ld, eps, xn, (uint8_t*)q8k,
                                                                                                  q8k_stride);
    Q38B_CUDA(ctx, cudaGetLastError());
    return Q38B_OK;
}

int q38b_gemv_bf16(q38b_ctx* ctx, const void* W_bf16, int K, int N, const float* x, float* y, void* stream) {
    if (!ctx || !W_bf16 || !x || !y || K <= 0 || K % 8 || N < 1) return Q38B_ERR_ARG;
    if (((uintptr_t)W_bf16 & 15) || ((uintptr_t)x & 15) || ((uintptr_t)y & 3)) return Q38B_ERR_ALIGN;
    gemv_bf16_kernel<<<(unsigned)N, BF16_THREADS, 0, (cudaStream_t)stream>>>((const uint16_t*)W_bf16, K, N, x, y);
    Q38B_CUDA(ctx, cudaGetLastError());
    return Q38B_OK;
}

int q38b_topk(q38b_ctx* ctx, const float* logits, long long ld, int n, int n_rows, int k, int index_offset, float* vals, int* idx, int out_ld,
              void* stream) {
    if (!ctx || !logits || !vals || !idx || n < 1 || n_rows < 1 || n_rows > 8 || k < 1 || k > TOPK_MAX_K || out_ld < k) return Q38B_ERR_ARG;
    if (n_rows > 1 && ld < n) return Q38B_ERR_ARG;
    const int n_chunks = (n + TOPK_CHUNK - 1) / TOPK_CHUNK;
    if (n_chunks > TOPK_MAX_CHUNKS) return Q38B_ERR_UNSUPPORTED;
    if (((uintptr_t)logits & 3) || ((uintptr_t)vals & 3) || ((uintptr_t)idx & 3)) return Q38B_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    TopkPair* lists = (TopkPair*)ctx->d_topk;
    auto lists_kernel = k <= TOPK_FEW ? topk_lists_kernel<true> : topk_lists_kernel<false>;
    lists_kernel<<<dim3((unsigned)((n_chunks + TOPK_STAGE1_WARPS - 1) / TOPK_STAGE1_WARPS), (unsigned)n_rows), TOPK_STAGE1_WARPS * 32, 0, st>>>(
        logits, ld, n, k, lists, n_chunks);
    if (k <= TOPK_FEW) {
        const int warps = (n_chunks * k + 32 * TOPK_FEW_ROUNDS - 1) / (32 * TOPK_FEW_ROUNDS);
        topk_merge_few_kernel<<<(unsigned)n_rows, 32 * warps, 0, st>>>(lists, n_chunks, k, logits, ld, index_offset, vals, idx, (long long)out_ld);
    } else {
        auto merge = n_chunks * k <= 8 * TOPK_MERGE_THREADS ? topk_merge_kernel<8> : topk_merge_kernel<TOPK_MAX_ROUNDS>;
        merge<<<(unsigned)n_rows, TOPK_MERGE_THREADS, 0, st>>>(lists, n_chunks, k, logits, ld, index_offset, vals, idx, (long long)out_ld);
    }
    Q38B_CUDA(ctx, cudaGetLastError());
    return Q38B_OK;
}

int q38b_swiglu_rows_inplace(q38b_ctx* ctx, float* G, const float* U, int B, int n, long long ld, int out_kind, void* stream) {
    if (!ctx || !G || !U || B < 1 || n <= 0 || n % 8 || ld < n || ld % 4) return Q38B_ERR_ARG;
    if (out_kind != Q38B_OUT_F16 && out_kind != Q38B_OUT_BF16) return Q38B_ERR_ARG;
    if (((uintptr_t)G & 15) || ((uintptr_t)U & 15)) return Q38B_ERR_ALIGN;
    const int smem = 2 * n;
    if (smem > ctx->smem_optin) return Q38B_ERR_NOMEM;
    cudaStream_t st = (cudaStream_t)stream;
    const int threads = swiglu_rows_threads(n);
    const bool bf = out_kind == Q38B_OUT_BF16;
    auto kern = threads == 512 ? (bf ? swiglu_rows_inplace_kernel<true, 512> : swiglu_rows_inplace_kernel<false, 512>)
              : threads == 256 ? (bf ? swiglu_rows_inplace_kernel<true, 256> : swiglu_rows_inplace_kernel<false, 256>)
                               : (bf ? swiglu_rows_inplace_kernel<true, 128> : swiglu_rows_inplace_kernel<false, 128>);
    const int rc = q38b_ensure_kernel_smem(ctx, (const void*)kern, ctx->smem_optin, false);
    if (rc != Q38B_OK) return rc;
    kern<<<(unsigned)B, (unsigned)threads, smem, st>>>(G, U, n, ld);
    Q38B_CUDA(ctx, cudaGetLastError());
    return Q38B_OK;
}

int q38b_gemv_q8k(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int M, const void* q8k,
                  long long q8k_stride, int nb, float* y, long long y_ld, int accumulate, void* stream) {
    return q38b_gemv_q8k_scatter(ctx, type, W, row_bytes, K, M, q8k, q8k_stride, nb, y, y_ld, accumulate, nullptr, 0, stream);
}

// one matrix, columns of Q8_K blocks
static ColsCall cols_call(uint32_t type, const void* W, size_t row_bytes, int K, int M, const void* q8k, long long q8k_stride, int nb, float* y, long long y_ld,
                          int accumulate, float* const* y_peers, int n_peers) {
    ColsCall c;
    c.type = type;
    c.row_bytes = row_bytes;
    c.K = K;
    c.nb = nb;
    c.n_mats = 1;
    c.W[0] = W;
    c.M[0] = M;
    c.y[0] = y;
    c.y_ld[0] = y_ld;
    c.xq = q8k;
    c.xq_ld = q8k_stride * Q8K_BYTES;
    c.accumulate = accumulate ? 1 : 0;
    c.y_peers = y_peers;
    c.n_peers = n_peers;
    return c;
}

// the columns of `c` on the one-column kernel's granules (p: their plan)
static int granule_launch(q38b_ctx* ctx, Plan1& p, const ColsCall& c, cudaStream_t st) {
    Gemv1Args& g = p.a;
    for (int i = 0; i < c.n_mats; i++) {
        (i == 0 ? g.W : g.W_more[i - 1]) = (const uint8_t*)c.W[i];
        (i == 0 ? g.y : g.y_more[i - 1]) = c.y[i];
        (i == 0 ? g.y_ld : g.y_ld_more[i - 1]) = c.y_ld[i];
        (i == 0 ? g.M : g.M_more[i - 1]) = c.M[i];
        for (int pr = 0; pr < c.n_peers; pr++) (i == 0 ? g.y_peer[pr] : g.y_peer_more[i - 1][pr]) = c.y_peers[i * c.n_peers + pr];
    }
    g.row_bytes = (long long)c.row_bytes;
    g.xq = (const uint8_t*)c.xq;
    g.xq_ld = c.xq_ld;
    g.x_f32 = c.x_f32;
    g.xf_ld = c.x_f32 ? c.x_f32_ld : c.xd32_ld;
    g.xd32 = c.xd32;
    g.n_peers = c.n_peers;
    g.static_weights = ctx->static_weights;
    g.status = ctx->d_status;
    g.codebook = q38b_grid_source(ctx, c.type);
    g.K = c.K;
    g.accumulate = c.accumulate;
    return dispatch_gemv1(ctx, c.type, p, st);
}

int q38b_gemv_q8k_scatter(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int M, const void* q8k,
                          long long q8k_stride, int nb, float* y, long long y_ld, int accumulate, float* const* y_peers,
                          int n_peers, void* stream) {
    if (!ctx || !W || !q8k || !y) return Q38B_ERR_ARG;
    if (n_peers < 0 || n_peers > 7 || (n_peers > 0 && !y_peers)) return Q38B_ERR_ARG;
    for (int i = 0; i < n_peers; i++) if (!y_peers[i] || ((uintptr_t)y_peers[i] & 3)) return Q38B_ERR_ARG;
    if (!known_format(type)) return Q38B_ERR_UNSUPPORTED;
    if (K <= 0 || K % 256 || M < 1 || nb < 1 || nb > 8 || y_ld < M || q8k_stride < K / 256) return Q38B_ERR_ARG;
    if (row_bytes < q38b_row_bytes(type, K)) return Q38B_ERR_ARG;
    const int al = format_alignment(type);
    if (((uintptr_t)W & 15) || (row_bytes % al) || ((uintptr_t)q8k & 3) || ((uintptr_t)y & 3)) return Q38B_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    if (nb > 1 && !q38b_cols_in_parts(type, K)) {
        // every column is what a launch of its own would give (but for the row groups of IQ3_XXS, a single column's)
        for (int c = 0; c < nb;) {
            Plan1 p1;
            bool granule;
            const int n = next_launch(ctx, type, K, &M, 1, row_bytes, nb - c, false, &granule, &p1);
            const uint8_t* xq = (const uint8_t*)q8k + (size_t)c * q8k_stride * Q8K_BYTES;
            float* peers_c[7];
            for (int i = 0; i < n_peers; i++) peers_c[i] = y_peers[i] + (size_t)c * y_ld;
            const ColsCall call = cols_call(type, W, row_bytes, K, M, xq, q8k_stride, n, y + (size_t)c * y_ld, y_ld, accumulate, peers_c, n_peers);
            const int rc = granule ? granule_launch(ctx, p1, call, st)
                         : n == 1 ? q38b_gemv_q8k_scatter(ctx, type, W, row_bytes, K, M, xq, q8k_stride, 1, y + (size_t)c * y_ld, y_ld, accumulate, peers_c, n_peers, stream)
                                  : q38b_cols_launch(ctx, call, stream);
            if (rc != Q38B_OK) return rc;
            c += n;
        }
        return Q38B_OK;
    }
    if (nb == 1 && (!ctx->uniform_columns || one_column_only((int)type))) {
        // single column: the dp4a kernel (one lane per 32- or 64-weight granule)
        Plan1 p1;
        memset(&p1, 0, sizeof(p1));
        const int rc1 = plan_gemv1(ctx, type, K, &M, 1, row_bytes, &p1);
        if (rc1 == Q38B_OK) {
            Gemv1Args& g = p1.a;
            g.W = (const uint8_t*)W;
            g.row_bytes = (long long)row_bytes;
            g.xq = (const uint8_t*)q8k;
            g.x_f32 = nullptr;
            g.y = y;
            g.n_peers = n_peers;
            g.static_weights = ctx->static_weights;
            for (int i = 0; i < n_peers; i++) g.y_peer[i] = y_peers[i];
            g.status = ctx->d_status;
            g.codebook = q38b_grid_source(ctx, type);
            g.K = K;
            g.M = M;
            g.accumulate = accumulate ? 1 : 0;
            return dispatch_gemv1(ctx, type, p1, st);
        }
    }
    // more (tile, K-part) sums than the scratch area holds: one launch per block of rows
    const long long rows_per_launch = q38b_cols_max_rows(ctx, type, K);
    if (rows_per_launch > 0 && M > rows_per_launch) {
        for (long long m0 = 0; m0 < M; m0 += rows_per_launch) {
            const int m = (int)std::min<long long>(rows_per_launch, M - m0);
            float* peers_at[7];
            for (int i = 0; i < n_peers; i++) peers_at[i] = y_peers[i] + m0;
            const int rc = q38b_gemv_q8k_scatter(ctx, type, (const uint8_t*)W + (size_t)m0 * row_bytes, row_bytes, K, m, q8k, q8k_stride, nb, y + m0,
                                                 y_ld, accumulate, n_peers ? peers_at : nullptr, n_peers, stream);
            if (rc != Q38B_OK) return rc;
        }
        return Q38B_OK;
    }
    return q38b_cols_launch(ctx, cols_call(type, W, row_bytes, K, M, q8k, q8k_stride, nb, y, y_ld, accumulate, y_peers, n_peers), stream);
}

static bool gemvn_group_args(const q38b_ctx* ctx, uint32_t type, int n_mats, size_t row_bytes, int K, int nb) {
    if (!ctx || n_mats < 1 || n_mats > G1_MAX_MATS || !known_format(type) || K <= 0 || K % 256 || nb < 1 || nb > 8) return false;
    return row_bytes >= q38b_row_bytes(type, K) && !(one_column_only((int)type) && nb == 1);
}

int q38b_gemvn_group_plannable(const q38b_ctx* ctx, uint32_t type, int n_mats, size_t row_bytes, int K, const int* M, int nb) {
    return gemvn_group_args(ctx, type, n_mats, row_bytes, K, nb) && q38b_cols_take(ctx, type, K, M, n_mats, row_bytes, nb, false) == nb;
}

int q38b_gemvn_group(q38b_ctx* ctx, uint32_t type, int n_mats, const void* const* W, size_t row_bytes, int K, const int* M,
                     const void* q8k, long long q8k_stride, int nb, float* const* y, const long long* y_ld, void* stream) {
    return q38b_gemvn_group_x(ctx, type, n_mats, W, row_bytes, K, M, q8k, q8k_stride, nullptr, 0, nb, y, y_ld, nullptr, 0, stream);
}

int q38b_gemvn_group_x(q38b_ctx* ctx, uint32_t type, int n_mats, const void* const* W, size_t row_bytes, int K, const int* M,
                       const void* q8k, long long q8k_stride, const float* x_f32, long long x_f32_ld, int nb, float* const* y,
                       const long long* y_ld, float* const* y_peers, int n_peers, void* stream) {
    if (!ctx || !W || !M || !y || !y_ld || (!q8k == !x_f32) || n_mats < 1 || n_mats > G1_MAX_MATS) return Q38B_ERR_ARG;
    if (n_peers < 0 || n_peers > 7 || (n_peers > 0 && !y_peers)) return Q38B_ERR_ARG;   // y_peers[i * n_peers + r]: peer r's copy of matrix i's output
    if (!gemvn_group_args(ctx, type, n_mats, row_bytes, K, nb)) return Q38B_ERR_UNSUPPORTED;
    const int al = format_alignment(type);
    if (row_bytes % al) return Q38B_ERR_ALIGN;
    if (q8k && (((uintptr_t)q8k & 3) || q8k_stride < K / 256)) return Q38B_ERR_ALIGN;
    if (x_f32 && (((uintptr_t)x_f32 & 15) || x_f32_ld < K || x_f32_ld % 4)) return Q38B_ERR_ALIGN;
    for (int i = 0; i < n_mats; i++) {
        if (!W[i] || !y[i] || M[i] < 1 || y_ld[i] < M[i]) return Q38B_ERR_ARG;
        if (((uintptr_t)W[i] & 15) || ((uintptr_t)y[i] & 3)) return Q38B_ERR_ALIGN;
    }
    ColsCall c;
    c.type = type;
    c.row_bytes = row_bytes;
    c.K = K;
    c.nb = nb;
    c.n_mats = n_mats;
    for (int i = 0; i < n_mats; i++) {
        c.W[i] = W[i];
        c.M[i] = M[i];
        c.y[i] = y[i];
        c.y_ld[i] = y_ld[i];
    }
    c.xq = q8k;
    c.xq_ld = q8k_stride * Q8K_BYTES;
    c.x_f32 = x_f32;
    c.x_f32_ld = x_f32_ld;
    c.y_peers = y_peers;
    c.n_peers = n_peers;
    Plan1 p1;
    long long rows = 0;
    for (int i = 0; i < n_mats; i++) rows += M[i];
    if (nb >= 2 && nb <= G1_COLS && cols_by_granule(ctx, type, rows, K / 256, nb, false) && plan_gemv1_cols(ctx, type, K, M, n_mats, row_bytes, nb, false, &p1) == Q38B_OK)
        return granule_launch(ctx, p1, c, (cudaStream_t)stream);
    const int rc = q38b_cols_launch(ctx, c, stream);
    return rc == Q38B_ERR_NOMEM ? Q38B_ERR_UNSUPPORTED : rc;
}

int q38b_gemv_group_plannable(const q38b_ctx* ctx, uint32_t type, int n_mats, size_t row_bytes, int K, const int* M) {
    if (!ctx || ctx->uniform_columns || n_mats < 1 || n_mats > G1_MAX_MATS || !known_format(type) || K <= 0 || K % 256) return 0;
    Plan1 p1;
    return plan_gemv1(ctx, type, K, M, n_mats, row_bytes, &p1) == Q38B_OK;
}

// Test hook: the one-column kernel's plan on a 148-SM device as CTAs per SM * 100000 + one-copy tiles * 10000 + rows per
// tile * 100 + stages (0: the shape does not fit it).
int q38b_debug_gemv1_rows(uint32_t type, int K, int M, size_t row_bytes, int rowgroup, int one_cta) {
    q38b_ctx ctx;
    ctx.sm_count = 148;
    ctx.smem_optin = 232448;
    ctx.rowgroup = rowgroup;
    ctx.one_cta = one_cta;
    Plan1 p1;
    if (!known_format(type) || K <= 0 || K % 256 || plan_gemv1(&ctx, type, K, &M, 1, row_bytes, &p1) != Q38B_OK) return 0;
    return p1.occ * 100000 + p1.a.contiguous * 10000 + p1.rows * 100 + p1.a.n_stages;
}

// Test hook: how many of `left` columns the next launch of the one-column kernel takes on such a device.
int q38b_debug_gemv1_cols(uint32_t type, int K, int M, size_t row_bytes, int left) {
    q38b_ctx ctx;
    ctx.sm_count = 148;
    ctx.smem_optin = 232448;
    Plan1 p1;
    return known_format(type) && K > 0 && K % 256 == 0 && left >= 1 ? next_cols(&ctx, type, K, M, row_bytes, left, &p1) : 0;
}

// Test hook: two to four columns by granules never (1), wherever there is a plan (2), by the rule (0)
int q38b_debug_set_cols_route(q38b_ctx* ctx, int mode) {
    if (!ctx || mode < 0 || mode > 2) return Q38B_ERR_ARG;
    ctx->cols_route = mode;
    return Q38B_OK;
}

int q38b_gemv_group(q38b_ctx* ctx, uint32_t type, int n_mats, const void* const* W, size_t row_bytes, int K, const int* M,
                    const void* q8k, const float* x_f32, float* const* y, void* stream) {
    return q38b_gemv_group_peers(ctx, type, n_mats, W, row_bytes, K, M, q8k, x_f32, y, nullptr, 0, stream);
}

int q38b_gemv_group_peers(q38b_ctx* ctx, uint32_t type, int n_mats, const void* const* W, size_t row_bytes, int K, const int* M,
                          const void* q8k, const float* x_f32, float* const* y, float* const* y_peers, int n_peers, void* stream) {
    if (!ctx || !W || !M || !y || n_mats < 1 || n_mats > G1_MAX_MATS || (!q8k == !x_f32)) return Q38B_ERR_ARG;
    if (n_peers < 0 || n_peers > 7 || (n_peers > 0 && !y_peers)) return Q38B_ERR_ARG;
    for (int i = 0; i < n_mats * n_peers; i++) if (!y_peers[i] || ((uintptr_t)y_peers[i] & 3)) return Q38B_ERR_ARG;
    if (!known_format(type)) return Q38B_ERR_UNSUPPORTED;
    if (K <= 0 || K % 256 || row_bytes < q38b_row_bytes(type, K)) return Q38B_ERR_ARG;
    const int al = format_alignment(type);
    if ((row_bytes % al) || (q8k && ((uintptr_t)q8k & 3)) || (x_f32 && ((uintptr_t)x_f32 & 15))) return Q38B_ERR_ALIGN;
    for (int i = 0; i < n_mats; i++) {
        if (!W[i] || !y[i] || M[i] < 1) return Q38B_ERR_ARG;
        if (((uintptr_t)W[i] & 15) || ((uintptr_t)y[i] & 3)) return Q38B_ERR_ALIGN;
    }
    if (ctx->uniform_columns) return Q38B_ERR_UNSUPPORTED;
    Plan1 p1;
    memset(&p1, 0, sizeof(p1));
    if (plan_gemv1(ctx, type, K, M, n_mats, row_bytes, &p1) != Q38B_OK) return Q38B_ERR_UNSUPPORTED;   // shapes only the tensor-core kernel takes
    Gemv1Args& g = p1.a;
    g.W = (const uint8_t*)W[0];
    g.y = y[0];
    g.M = M[0];
    for (int i = 1; i < n_mats; i++) {
        g.W_more[i - 1] = (const uint8_t*)W[i];
        g.y_more[i - 1] = y[i];
        g.M_more[i - 1] = M[i];
    }
    g.row_bytes = (long long)row_bytes;
    g.xq = (const uint8_t*)q8k;
    g.x_f32 = x_f32;
    g.sync = take_pending_sync(ctx);
    g.n_peers = n_peers;
    for (int i = 0; i < n_mats; i++)
        for (int pr = 0; pr < n_peers; pr++) (i == 0 ? g.y_peer[pr] : g.y_peer_more[i - 1][pr]) = y_peers[i * n_peers + pr];
    g.static_weights = ctx->static_weights;
    g.status = ctx->d_status;
    g.codebook = q38b_grid_source(ctx, type);
    g.K = K;
    g.accumulate = 0;
    cudaStream_t st = (cudaStream_t)stream;
    return dispatch_gemv1(ctx, type, p1, st);
}

int q38b_quantize_act_q8(q38b_ctx* ctx, const float* x, int K, int n_rows, int8_t* q, float* d, float* s, void* stream) {
    if (!ctx || !x || !q || !d || !s || K <= 0 || K % 32 || n_rows < 1) return Q38B_ERR_ARG;
    if (((uintptr_t)x | (uintptr_t)d | (uintptr_t)s) & 3) return Q38B_ERR_ALIGN;
    const long long blocks = (long long)n_rows * (K / 32);
    quantize_act_q8_kernel<<<(unsigned)((blocks + ACT_WARPS - 1) / ACT_WARPS), ACT_WARPS * 32, 0, (cudaStream_t)stream>>>(x, blocks, q, d, s);
    Q38B_CUDA(ctx, cudaGetLastError());
    return Q38B_OK;
}

int q38b_gemv_act_q8(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int M, const int8_t* q, const float* d,
                     int nb, int act_ld, float* y, int y_ld, int accumulate, void* stream) {
    if (!ctx || !W || !q || !d || !y) return Q38B_ERR_ARG;
    if (!known_format(type)) return Q38B_ERR_UNSUPPORTED;
    if (K <= 0 || K % 256 || M < 1 || nb < 1 || nb > 8 || y_ld < M || act_ld < K || act_ld % 32) return Q38B_ERR_ARG;
    if (row_bytes < q38b_row_bytes(type, K)) return Q38B_ERR_ARG;
    const int al = format_alignment(type);
    if (((uintptr_t)W & 15) || (row_bytes % al) || ((uintptr_t)q & 3) || (act_ld & 3) || ((uintptr_t)d & 3) || ((uintptr_t)y & 3)) return Q38B_ERR_ALIGN;
    // The one-column kernel on its lane-per-granule mapping, or several columns a launch with the same arithmetic: every
    // column is the single-column result (the promise of src/cuda/gemv.cuh:31-34 of the reference).
    const int saved_rg = ctx->rowgroup;
    ctx->rowgroup = 0;
    int rc = Q38B_OK;
    for (int c = 0; c < nb && rc == Q38B_OK;) {
        Plan1 p;
        bool granule;
        const int n = next_launch(ctx, type, K, &M, 1, row_bytes, nb - c, true, &granule, &p);
        ColsCall call = cols_call(type, W, row_bytes, K, M, q + (size_t)c * act_ld, 0, n, y + (size_t)c * y_ld, y_ld, accumulate, nullptr, 0);
        call.xq_ld = act_ld;
        call.xd32 = d + (size_t)c * (act_ld / 32);
        call.xd32_ld = act_ld / 32;
        if (n > 1 && !granule) {
            rc = q38b_cols_launch(ctx, call, stream);
            c += n;
            continue;
        }
        if (n == 1) {
            memset(&p, 0, sizeof(p));
            const bool fits_one = ctx->one_cta && type != T_Q8_0 && plan_gemv1_rows(ctx, type, K, &M, 1, row_bytes, 8, 1, 1, gridx_copies((int)type) > 0, &p) == Q38B_OK;
            if (!fits_one || !act_q8_one_cta(ctx, type, p)) {
                Plan1 two;
                const int saved_one = ctx->one_cta;
                ctx->one_cta = 0;
                const bool fits_two = plan_gemv1(ctx, type, K, &M, 1, row_bytes, &two) == Q38B_OK;
                ctx->one_cta = saved_one;
                if (fits_two) p = two;
                else if (!fits_one) { rc = Q38B_ERR_NOMEM; break; }
            }
        }
        rc = granule_launch(ctx, p, call, (cudaStream_t)stream);
        c += n;
    }
    ctx->rowgroup = saved_rg;
    return rc;
}

int q38b_gemv_f32(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int M, const float* x, long long x_ld,
                  int nb, float* y, long long y_ld, int accumulate, void* q8k_scratch, size_t scratch_bytes, void* stream) {
    if (!ctx || !x || !q8k_scratch || nb < 1 || nb > 8 || K <= 0 || K % 256) return Q38B_ERR_ARG;
    if (scratch_bytes < (size_t)nb * q38b_q8k_bytes(K)) return Q38B_ERR_NOMEM;
    int rc = q38b_quantize_q8k(ctx, x, x_ld, K, nb, q8k_scratch, K / 256, stream);
    if (rc != Q38B_OK) return rc;
    return q38b_gemv_q8k(ctx, type, W, row_bytes, K, M, q8k_scratch, K / 256, nb, y, y_ld, accumulate, stream);
}

}  // extern "C"
