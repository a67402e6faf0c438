// q38b_gemvn.cu -- launch planning of the several-column matvec (q38b_gemv.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
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

// How many different words the lanes of a decoder's main load want from the bank that most of them meet on, rows `pitch` bytes apart
// (a 64-bit load is served half a warp, four rows, at a time).
int bank_degree(uint32_t type, int pitch) {
    int bytes, step;   // of a lane's load, and between the four lanes of a row
    switch (type) {
        case T_Q4_K: case T_Q5_K: bytes = step = 8; break;
        case T_IQ4_XS: case T_Q2_K: bytes = step = 4; break;
        case T_Q8_0: bytes = 2; step = 8; break;
        case T_Q6_K: bytes = 2; step = 4; break;
        case T_IQ3_XXS: case T_IQ3_S: case T_IQ2_XS: bytes = step = 2; break;
        default: bytes = step = 1; break;
    }
    int want[32] = {}, most = 1;
    int seen[64], n = 0;
    for (int g = 0; g < (bytes == 8 ? 4 : 8); g++)
        for (int b = 0; b < 4 * step; b += std::max(4, step == 8 && bytes == 2 ? 8 : 4)) {
            const int w = (g * pitch + b) / 4;
            bool had = false;
            for (int i = 0; i < n; i++) had |= seen[i] == w;
            if (had) continue;
            seen[n++] = w;
            most = std::max(most, ++want[w % 32]);
        }
    return most;
}
// a 64-bit load wants the rows an odd multiple of 32 bytes apart, the others of 16
int padded_pitch(uint32_t type, int bytes) {
    const bool wide = type == T_Q4_K || type == T_Q5_K || type == T_Q8_0;
    int pitch = align_up(bytes, 16);
    while (wide ? pitch % 64 != 32 : pitch % 32 != 16) pitch += 16;
    return pitch;
}

struct Plan {
    GemvArgs a;
    int grid;
    int smem;
    double rating;   // of the division: the share of the launch left to the decoders
};

int table_bytes(uint32_t type) {
    return type == T_IQ3_XXS ? 1024 << cb1_rep_log2(T_IQ3_XXS) : type == T_IQ3_S ? 2048 << cb1_rep_log2(T_IQ3_S) : gridx_bytes((int)type);
}

// Carves up the shared memory of one CTA: barriers | activation scales | activations | zeros | tables | unit sums | ring.
//
// How a tile's row is divided: into chunks of chunk_sb super-blocks (a stage each), a chunk into units of one, two or four
// super-blocks, the units among kw warps; rows with few units leave warps for further groups, each with tiles of its own.  A
// division is rated by the share of the launch that it leaves to the decoders:
//   * units on the warps: work / (rounds of the warps), each unit with a fixed cost of 0.55 of a super-block;
//   * nine warps and more keep the schedulers busy, as long as each scheduler has as many of them: 12 warps beat 18 (17408 x 2816
//     IQ3_S, 3 x 4 warps 16.1 us, 6 x 3 17.5); of a last round of tiles that some groups sit out about half is lost, the others
//     being faster meanwhile (6144 x 5120 IQ2_S, 2.6 tiles a CTA: two groups 13.4 us, one 14.3);
//   * a copy costs the copy engine its bytes and 300 more;
//   * one copy of 16 packed rows a stage loses 18 % to a copy per padded row (its rows meet on banks, and nothing of the stage can be
//     read before all of it is there), and 4 % for every further row that meets on a bank: 17408 x 5120 Q8_0, seven columns, whose
//     rows all meet in twos on two banks, 39.1 us in one copy, 27.0 in sixteen.  It is for rows of a few hundred bytes.
// How far the ring runs ahead has no term: any two stages a group are enough.  Measured over all divisions of 593 shapes (thirteen
// formats, 5120 and 17408 rows of 1024 to 17408 weights, two to eight columns, Q8_K and per-32) the division picked takes 1.2 % more
// than the best on average and 18 % at most; rated by bytes under way, as before, it took 4.9 % more on average and 56 % at most.
// With 356 shapes of 1024 to 12288 rows it is 1.6 % and 23 %.
constexpr double UNIT_COST = 0.55, BUSY_WARPS = 9.0, COPY_BYTES = 300.0, ONE_COPY = 0.82, PER_ROW_MEETING = 0.04;
int search_plan(const q38b_ctx* ctx, uint32_t type, int K, const int* Ms, int n_mats, size_t row_bytes, int nb, bool a32, Plan* p) {
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
    const long long items = (long long)a.n_tiles * a.n_parts;
    p->grid = (int)std::max<long long>(1, std::min<long long>(ctx->sm_count, items));
    // a CTA's range of (part, tile) items touches at most two neighbouring parts: it stages their activations only
    a.act_sb = a.n_parts == 1 ? nsb : std::min(nsb, 2 * a.item_sb);
    a.off_actd = GEMV_HEADER;
    a.off_actq = a.off_actd + a.act_sb * (a32 ? 256 : 32);
    a.off_bsum = align_up(a.off_actq + nb * (a.act_sb * 256 + act_skew((int)type)), 16);
    a.off_zero = align_up(a.off_bsum + a.act_sb * 8 * bsum_bytes((int)type, a32), 128);
    a.off_cb = a.off_zero + (wants_zeros((int)type) ? 384 : 0);
    a.off_sgn = a.off_cb + align_up(table_bytes(type), 128);
    a.off_red = a.off_sgn + (sign_table((int)type) ? 128 * 8 * SIGN_COPIES : 0);
    const int packed = nsb * bb;
    const bool packed_rows = a.n_parts == 1 && (long long)row_bytes == packed;
    const double one_copy_worth = packed_rows ? ONE_COPY / (1.0 + PER_ROW_MEETING * (bank_degree(type, packed) - 1)) : 0.0;
    const double cta_items = (double)items / p->grid;
    p->rating = 0.0;
    for (int unit = 1; unit <= 4; unit *= 2)
        for (int n_chunks = 1; n_chunks <= (p->rating > 0.0 ? std::min(a.item_sb, 12) : a.item_sb); n_chunks++) {
            const int cs = std::min(a.item_sb, ((a.item_sb + n_chunks - 1) / n_chunks + unit - 1) / unit * unit);
            if ((a.item_sb + cs - 1) / cs != n_chunks) continue;
            const int slots = (a.item_sb + unit - 1) / unit, units = (cs + unit - 1) / unit;
            const int least_rounds = (units + GEMV_MAX_WARPS - 1) / GEMV_MAX_WARPS;
            for (int one_copy = n_chunks == 1 && packed_rows ? 1 : 0; one_copy >= 0; one_copy--) {
                const int pitch = one_copy ? packed : padded_pitch(type, cs * bb + 32);
                const int stage = align_up(TILE_ROWS * pitch + 64, 128);
                if (a.off_red + 2 * stage > budget) continue;
                const double copy = one_copy ? (double)TILE_ROWS * packed : (double)cs * bb;
                const double copied = copy / (copy + COPY_BYTES) * (one_copy ? one_copy_worth : 1.0);
                for (int rounds = least_rounds; rounds <= std::min(units, least_rounds + 5); rounds++) {
                    const int kw = (units + rounds - 1) / rounds;
                    const double rows = copied * a.item_sb / ((double)n_chunks * rounds * kw * (unit + UNIT_COST));
                    if (rows <= p->rating) continue;
                    for (int groups = n_chunks == 1 ? GEMV_MAX_WARPS / kw : 1; groups >= 1; groups--) {
                        const int off_stage = align_up(a.off_red + groups * GEMV_TILEBUF * slots * 64 * a.cols, 128);
                        const int stages = std::min(GEMV_MAX_STAGES, (budget - off_stage) / stage) / groups * groups;
                        if (stages < 2 * groups) continue;
                        const int warps = kw * groups;
                        const double busy = std::min(1.0, warps / BUSY_WARPS) * warps / ((warps + 3) / 4 * 4);
                        const double turns = cta_items / groups;
                        const double rating = rows * busy * (a.n_parts == 1 ? std::sqrt(turns / std::ceil(turns)) : 1.0);
                        if (rating <= p->rating) continue;
                        p->rating = rating;
                        a.contiguous = one_copy;
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
                }
            }
        }
    return p->rating > 0.0 ? Q38B_OK : Q38B_ERR_NOMEM;
}

// The search takes some 2.7 us of a call whose launch takes about as much, and depends on nothing but these numbers: each thread keeps
// the plans of the last shapes it met (a layer has four to seven).
struct PlanKey {
    size_t row_bytes;
    long long part_items;
    uint32_t type;
    int K, nb, a32, n_mats, M[GEMV_MAX_MATS], sm_count, smem_optin;
};
int plan_gemv(const q38b_ctx* ctx, uint32_t type, int K, const int* Ms, int n_mats, size_t row_bytes, int nb, bool a32, Plan* p) {
    struct Entry { PlanKey key; Plan plan; int rc; bool used; };
    constexpr int ENTRIES = 32;
    static thread_local Entry kept[ENTRIES];
    PlanKey k;
    memset(&k, 0, sizeof(k));
    k.row_bytes = row_bytes;
    k.part_items = ctx->part_items;
    k.type = type;
    k.K = K;
    k.nb = nb;
    k.a32 = a32 ? 1 : 0;
    k.n_mats = n_mats;
    for (int i = 0; i < n_mats; i++) k.M[i] = Ms[i];
    k.sm_count = ctx->sm_count;
    k.smem_optin = ctx->smem_optin;
    uint64_t h = (uint64_t)row_bytes * 31 + type;
    for (int v : {K, nb, k.a32, k.M[0], k.M[1], k.M[2]}) h = (h ^ (uint64_t)v) * 0x9E3779B97F4A7C15ull;
    Entry& e = kept[(h >> 32) % ENTRIES];
    if (!e.used || memcmp(&e.key, &k, sizeof(k)) != 0) {
        e.rc = search_plan(ctx, type, K, Ms, n_mats, row_bytes, nb, a32, &e.plan);
        e.key = k;
        e.used = true;
    }
    *p = e.plan;
    return e.rc;
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

bool q38b_cols_in_parts(uint32_t type, int K) { return part_count(type, K, false) > 1; }

long long q38b_cols_max_rows(const q38b_ctx* ctx, uint32_t type, int K) {
    const int parts = part_count(type, K, false);
    return parts == 1 ? 0 : ctx->part_items / parts * TILE_ROWS;
}

// A launch's time goes with about the 0.42nd power of its plan's rating down (5120 x 17408 IQ3_XXS, per-32: six columns at 0.213 47 us,
// four at 0.473 34, seven at 0.048 92), so that all columns at once lose to two halves from a rating of a fifth of the halves' on:
// there a long row's activations leave the ring two small stages that feed a few warps.
int q38b_cols_take(const q38b_ctx* ctx, uint32_t type, int K, const int* M, int n_mats, size_t row_bytes, int left, bool a32) {
    if (a32 && type == T_Q6_K) return 0;
    Plan all, half;
    int n = std::min(8, left);
    bool fits = plan_gemv(ctx, type, K, M, n_mats, row_bytes, n, a32, &all) == Q38B_OK;
    while (n > 1 && (!fits || all.rating < 0.25)) {   // (no plan is rated above one and few above 0.8: others need no second look)
        const int h = (n + 1) / 2;
        const bool half_fits = plan_gemv(ctx, type, K, M, n_mats, row_bytes, h, a32, &half) == Q38B_OK;
        if (fits && (!half_fits || all.rating >= 0.2 * half.rating)) break;
        n = h;
        fits = half_fits;
        all = half;
    }
    return fits ? n : 0;
}

// Test hook (not in the public header): the division of a row for nb columns on a 148-SM device with 227 KB of shared memory a CTA, no
// device needed: warps of a tile, groups, super-blocks a stage, stages, whether a stage is one copy, thousandths of the rating.
extern "C" int q38b_debug_gemvn_plan(uint32_t type, int K, int M, size_t row_bytes, int nb, int a32, int* out) {
    q38b_ctx ctx;
    ctx.sm_count = 148;
    ctx.smem_optin = 232448;
    ctx.part_items = 131072;
    Plan p;
    const int rc = plan_gemv(&ctx, type, K, &M, 1, row_bytes, nb, a32 != 0, &p);
    if (rc != Q38B_OK) return rc;
    const int v[6] = {p.a.kw, p.a.groups, p.a.chunk_sb, p.a.n_stages, p.a.contiguous, (int)(1000.0 * p.rating)};
    memcpy(out, v, sizeof(v));
    return Q38B_OK;
}
extern "C" int q38b_debug_gemvn_take(uint32_t type, int K, int M, size_t row_bytes, int left, int a32) {
    q38b_ctx ctx;
    ctx.sm_count = 148;
    ctx.smem_optin = 232448;
    ctx.part_items = 131072;
    return q38b_cols_take(&ctx, type, K, &M, 1, row_bytes, left, a32 != 0);
}

int q38b_cols_launch(q38b_ctx* ctx, const ColsCall& c, void* stream) {
    Plan p;
    const int rc = plan_gemv(ctx, c.type, c.K, c.M, c.n_mats, c.row_bytes, c.nb, c.xd32 != nullptr, &p);
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
