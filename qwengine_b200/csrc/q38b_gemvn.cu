// q38b_gemvn.cu -- launch planning of the several-column matvec (q38b_gemv.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "../../include/q38b200.h"
#include "q38b_gemv.cuh"
#include "q38b_internal.h"

using namespace q38b;

namespace {

constexpr int GEMV_WHOLE_ROW_K = 8192;          // longer rows run as K-parts (measured on B200: parts on K = 5120 / 6144 cost more per item than they even out)

int align_up(int v, int a) { return (v + a - 1) / a * a; }

// Rows that keep the one-column launch's bits are never cut into parts: their slices are added one after the other.
bool cut_into_parts(uint32_t type, int K, bool a32) { return K > GEMV_WHOLE_ROW_K && !a32 && !one_column_only((int)type); }
// super-blocks per K-part, at most: one per consumer warp, as long as two parts of activations for 8 columns and three stages of
// 16 rows fit
int part_most(uint32_t type) { return type == T_Q8_0 ? 10 : type == T_Q6_K || type == T_Q5_K ? 17 : GEMV_MAX_WARPS; }
int part_count(uint32_t type, int K, bool a32) {
    const int nsb = K / 256, most = part_most(type);
    return cut_into_parts(type, K, a32) ? std::min(GEMV_MAX_PARTS, (nsb + most - 1) / most) : 1;
}

// Whether at most two of the rows g of a tile, `pitch` bytes apart, meet on a bank when their four lanes each read `bytes` side by
// side (all eight rows with one load, four with a 64-bit load, which is served half a warp at a time).
bool few_conflicts(int pitch, int bytes) {
    int meet = 0;
    for (int k = 1; k < (bytes == 8 ? 4 : 8); k++) {
        const int d = k * pitch % 128;
        meet += d < 4 * bytes || 128 - d < 4 * bytes;
    }
    return meet <= 1;
}
// bytes a lane takes from its row with the decoder's main load
int lane_bytes(uint32_t type) {
    switch (type) {
        case T_Q4_K: case T_Q5_K: case T_Q8_0: return 8;
        case T_IQ4_XS: case T_Q6_K: case T_Q2_K: return 4;
        case T_IQ3_XXS: case T_IQ3_S: case T_IQ2_XS: return 2;
        default: return 1;
    }
}

struct Plan {
    GemvArgs a;
    int grid;
    int smem;
};

int table_bytes(uint32_t type) {
    return type == T_IQ3_XXS ? 1024 << cb1_rep_log2(T_IQ3_XXS) : type == T_IQ3_S ? 2048 << cb1_rep_log2(T_IQ3_S) : gridx_bytes((int)type);
}

// any: also a plan that leaves most warps without work.
// Carves up the shared memory of one CTA: barriers | activation scales | activations | zeros | tables | unit sums | ring.
int plan_gemv(const q38b_ctx* ctx, uint32_t type, int K, const int* Ms, int n_mats, size_t row_bytes, int nb, bool a32, bool any, Plan* p) {
    const int bb = block_bytes((int)type), nsb = K / 256;
    const int budget = ctx->smem_optin;
    GemvArgs& a = p->a;
    memset(p, 0, sizeof(*p));
    a.nsb = nsb;
    a.cols = (nb + 1) / 2 * 2;
    for (int i = 0; i < GEMV_MAX_MATS; i++) {
        a.tile_start[i] = a.n_tiles;
        if (i < n_mats) a.n_tiles += (Ms[i] + TILE_ROWS - 1) / TILE_ROWS;
    }
    for (int i = n_mats; i < GEMV_MAX_MATS; i++) a.tile_start[i] = a.n_tiles;
    // K-parts of about equal length.  A rule of K and the format alone, so that a sum is built from the same pieces
    // whatever the column count, the row count or the GPU count.
    a.n_parts = part_count(type, K, a32);
    for (int q = 0; q <= a.n_parts; q++) a.part_sb0[q] = (int)((long long)nsb * q / a.n_parts);
    for (int q = 0; q < a.n_parts; q++) a.item_sb = std::max(a.item_sb, a.part_sb0[q + 1] - a.part_sb0[q]);
    if (a.n_parts > 1 && (long long)a.n_tiles * a.n_parts > ctx->part_items) return Q38B_ERR_NOMEM;   // the scratch area's size
    // a CTA's range of (part, tile) items touches at most two neighbouring parts: it stages their activations only
    a.act_sb = a.n_parts == 1 ? nsb : std::min(nsb, 2 * a.item_sb);
    a.off_actd = GEMV_HEADER;
    a.off_actq = a.off_actd + a.act_sb * (a32 ? 256 : 32);
    a.off_bsum = align_up(a.off_actq + nb * (a.act_sb * 256 + act_skew((int)type)), 16);
    a.off_zero = align_up(a.off_bsum + a.act_sb * 8 * bsum_bytes((int)type, a32), 128);
    a.off_cb = a.off_zero + (wants_zeros((int)type) ? 384 : 0);
    a.off_sgn = a.off_cb + align_up(table_bytes(type), 128);
    a.off_red = a.off_sgn + (sign_table((int)type) ? 128 * 8 * SIGN_COPIES : 0);
    // How a tile's row is divided: into chunks of chunk_sb super-blocks (a stage each), a chunk into units of one, two or four
    // super-blocks, the units among kw warps; rows with few units leave warps for further groups, each with tiles of its own.
    // Rated by the share of the warps' time that is work (a unit's fixed cost counts as UNIT_COST of a super-block) and by the
    // bytes that the ring can have under way while a stage is being read.
    constexpr double UNIT_COST = 0.4;
    const int packed = nsb * bb, lb = lane_bytes(type);
    const bool packed_rows = a.n_parts == 1 && (long long)row_bytes == packed && few_conflicts(packed, lb);
    double best = 0.0;
    for (int unit = 1; unit <= 4; unit *= 2)
        for (int n_chunks = 1; n_chunks <= (best > 0.0 ? 4 : a.item_sb); n_chunks++) {
            const int cs = std::min(a.item_sb, ((a.item_sb + n_chunks - 1) / n_chunks + unit - 1) / unit * unit);
            if ((a.item_sb + cs - 1) / cs != n_chunks) continue;
            const bool one_copy = n_chunks == 1 && packed_rows;
            // rows an odd multiple of 16 bytes apart (32 for 64-bit loads) meet no bank
            int pitch = one_copy ? packed : align_up(cs * bb + 32, 16);
            while (!one_copy && (lb == 8 ? pitch % 64 != 32 : pitch % 32 != 16)) pitch += 16;
            const int stage = align_up(TILE_ROWS * pitch + 64, 128);
            if (a.off_red + 2 * stage > budget) continue;
            const int slots = (a.item_sb + unit - 1) / unit, units = (cs + unit - 1) / unit;
            const int copy = one_copy ? TILE_ROWS * packed : cs * bb;
            if (best > 0.0 && copy < 512) break;
            const int least_rounds = (units + GEMV_MAX_WARPS - 1) / GEMV_MAX_WARPS;
            for (int rounds = least_rounds; rounds <= std::min(units, least_rounds + 3); rounds++) {
                const int kw = (units + rounds - 1) / rounds;
                for (int groups = n_chunks == 1 ? GEMV_MAX_WARPS / kw : 1; groups >= 1; groups--) {
                    const int off_stage = align_up(a.off_red + groups * GEMV_TILEBUF * slots * 64 * a.cols, 128);
                    const int stages = std::min(GEMV_MAX_STAGES, (budget - off_stage) / stage) / groups * groups;
                    if (stages < 2 * groups) continue;
                    const double work = (double)a.item_sb / ((double)n_chunks * rounds * kw * (unit + UNIT_COST));
                    const double warps = std::min(1.0, (kw * groups + 4) / 24.0);
                    // bytes under way beside the stages being read, up to 48 KB; copies below 1.7 KB cost the copy engine's time
                    const double ring = std::min(1.0, (double)(stages - groups) * stage / (48.0 * 1024)) * std::min(1.0, copy / 1700.0);
                    const double score = work * warps * ring;
                    if (score > best * 1.0001) {
                        best = score;
                        a.contiguous = one_copy ? 1 : 0;
                        a.chunk_sb = cs;
                        a.unit_log2 = unit == 4 ? 2 : unit - 1;
                        a.kw = kw;
                        a.groups = groups;
                        a.slots = slots;
                        a.slot_stride = pitch;
                        a.stage_bytes = stage;
                        a.n_stages = stages;
                        a.off_stage = off_stage;
                        p->smem = off_stage + stages * stage;
                    }
                    break;   // fewer groups are worth less
                }
            }
        }
    if (best == 0.0) return Q38B_ERR_NOMEM;
    if (!any && a.kw * a.groups < std::min(8, (a.item_sb + 3) / 4)) return Q38B_ERR_NOMEM;   // fewer columns leave the ring room for chunks that feed the warps
    const long long items = (long long)a.n_tiles * a.n_parts;
    p->grid = (int)std::max<long long>(1, std::min<long long>(ctx->sm_count, items));
    return Q38B_OK;
}

template <int FMT, bool A32, bool PARTED>
int launch(q38b_ctx* ctx, const Plan& p, cudaStream_t st) {
    auto kern = gemv_kernel<FMT, A32, PARTED>;
    const int rc = q38b_ensure_kernel_smem(ctx, (const void*)kern, ctx->smem_optin, false);
    if (rc != Q38B_OK) return rc;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3(32 * (2 + GEMV_MAX_WARPS));
    cfg.dynamicSmemBytes = (size_t)p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p.a);
    if (e != cudaSuccess) { ctx->last_cuda = (int)e; return Q38B_ERR_CUDA; }
    return Q38B_OK;
}

template <int FMT>
int launch_format(q38b_ctx* ctx, const Plan& p, cudaStream_t st) {
    if (p.a.xd32) {
        if constexpr (FMT != T_Q6_K) return launch<FMT, true, false>(ctx, p, st);
        return Q38B_ERR_ARG;
    }
    if constexpr (!one_column_only(FMT)) {
        if (p.a.n_parts > 1) return launch<FMT, false, true>(ctx, p, st);
    }
    return launch<FMT, false, false>(ctx, p, st);
}

}  // namespace

long long q38b_cols_max_rows(const q38b_ctx* ctx, uint32_t type, int K) {
    const int parts = part_count(type, K, false);
    return parts == 1 ? 0 : ctx->part_items / parts * TILE_ROWS;
}

int q38b_cols_fit(const q38b_ctx* ctx, uint32_t type, int K, const int* M, int n_mats, size_t row_bytes, int nb, bool a32) {
    if (a32 && type == T_Q6_K) return 0;
    Plan p;
    int n = std::min(8, nb);
    while (n > 0 && plan_gemv(ctx, type, K, M, n_mats, row_bytes, n, a32, n == 1, &p) != Q38B_OK) n--;
    return n;
}

int q38b_cols_launch(q38b_ctx* ctx, const ColsCall& c, void* stream) {
    Plan p;
    const int rc = plan_gemv(ctx, c.type, c.K, c.M, c.n_mats, c.row_bytes, c.nb, c.xd32 != nullptr, true, &p);
    if (rc != Q38B_OK) return rc;
    GemvArgs& a = p.a;
    for (int i = 0; i < c.n_mats; i++) {
        (i == 0 ? a.W : a.W_more[i - 1]) = (const uint8_t*)c.W[i];
        (i == 0 ? a.y : a.y_more[i - 1]) = c.y[i];
        (i == 0 ? a.y_ld : a.y_ld_more[i - 1]) = c.y_ld[i];
        (i == 0 ? a.M : a.M_more[i - 1]) = c.M[i];
        for (int r = 0; r < c.n_peers; r++) (i == 0 ? a.y_peer[r] : a.y_peer_more[i - 1][r]) = c.y_peers[i * c.n_peers + r];
    }
    a.row_bytes = (long long)c.row_bytes;
    a.xq = (const uint8_t*)c.xq;
    a.xq_ld = c.xq_ld;
    a.x_f32 = c.x_f32;
    a.x_f32_ld = c.x_f32_ld;
    a.xd32 = c.xd32;
    a.xd32_ld = c.xd32_ld;
    a.n_peers = c.n_peers;
    a.static_weights = ctx->static_weights;
    a.status = ctx->d_status;
    a.codebook = q38b_grid_source(ctx, c.type);
    a.K = c.K;
    a.nb = c.nb;
    a.accumulate = c.accumulate;
    a.parts = ctx->d_parts;
    a.part_count = ctx->d_part_count;
    cudaStream_t st = (cudaStream_t)stream;
    switch (c.type) {
        case T_Q8_0: return launch_format<T_Q8_0>(ctx, p, st);
        case T_Q4_K: return launch_format<T_Q4_K>(ctx, p, st);
        case T_Q5_K: return launch_format<T_Q5_K>(ctx, p, st);
        case T_Q6_K: return launch_format<T_Q6_K>(ctx, p, st);
        case T_IQ3_XXS: return launch_format<T_IQ3_XXS>(ctx, p, st);
        case T_IQ3_S: return launch_format<T_IQ3_S>(ctx, p, st);
        case T_IQ4_XS: return launch_format<T_IQ4_XS>(ctx, p, st);
        case T_Q2_K: return launch_format<T_Q2_K>(ctx, p, st);
        case T_IQ2_XXS: return launch_format<T_IQ2_XXS>(ctx, p, st);
        case T_IQ2_XS: return launch_format<T_IQ2_XS>(ctx, p, st);
        case T_IQ2_S: return launch_format<T_IQ2_S>(ctx, p, st);
        case T_IQ1_S: return launch_format<T_IQ1_S>(ctx, p, st);
        case T_IQ1_M: return launch_format<T_IQ1_M>(ctx, p, st);
        default: return Q38B_ERR_UNSUPPORTED;
    }
}
