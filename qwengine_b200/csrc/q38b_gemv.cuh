// q38b_gemv.cuh -- the several-column matvec kernel: y[c][r] (+)= W[r,:] . x_c for 1..8 activation columns.
//
// Replaces k_gemv_q8 / gemv_q8n of the reference (src/cuda/gemv.cu:51-125, 215-228).  Shape of the kernel:
//   * persistent CTAs (one per SM): a producer warp, GEMV_MAX_WARPS warps of which as many consume as divide K well, and a warp that adds up tiles;
//   * the weight rows stream HBM -> shared memory through 1-D bulk (TMA) copies into ONE ring of stages, completion tracked by
//     mbarriers; a stage holds a 16-row tile (or a K-chunk of it); GGUF blocks of most formats are only 2-byte aligned, so
//     each copy moves the 16-byte aligned superset of its range and the consumers index from the remainder;
//   * the warps divide K: warp w of a tile's `kw` always takes the same super-blocks (one, two or four in a row, by the row's
//     length), decodes them into int8 mma fragments (q38b_decode.cuh) and keeps the 16 x 8 sums in registers.  All warps walk
//     the stages in order; per tile each puts its sums into its slot and arrives on the tile's mbarrier, and a further warp
//     adds the slots in order and stores the rows, so results do not depend on timing.  (The warps of a tile taking turns at
//     that held the tile's stage: 2 x 17408 x 5120 Q4_K, two columns, 26.3 us, 25.3 with a warp of its own.)  Short rows:
//     several groups of kw warps take tiles in turn;
//   * activations (int8 values and scales of all columns) and the tables are staged in shared memory once per CTA, the columns
//     32 (16) bytes off a multiple of 128, so that the four or eight columns of one load meet no bank;
//   * rows longer than 8192 are cut into K-parts of at most 20 super-blocks, Q5_K / Q6_K 17, Q8_0 10 (a rule of K and the format alone).  The work
//     items (part, tile), part-major, are dealt to the CTAs as equal contiguous ranges: a CTA then needs the
//     activations of at most two neighbouring parts, which leaves the shared memory to the weight stages, and 320
//     tiles of 68 super-blocks keep 148 SMs evenly busy instead of 24 of them working a second round.  A part's sums
//     go to a scratch area in global memory; the adding warp raises the tile's counter, looks at the count one item later
//     and, where it counted the last part, reads them all back, adds them in part order and stores the row sums --
//     the result does not depend on who computed what or when.  No fences and no waiting on other CTAs' progress: a scratch
//     slot rests at a NaN pattern no sum can have and is read until it holds sums that are already on their way.
// What bounds it: the decoders' instructions (see q38b_decode.cuh; an IMMA takes nine clocks from the integer units), then the
// prologue (two to seven columns of 5120 floats: 4,000 to 6,800 clocks a launch).  A copy costs the copy engine about 70 clocks
// whatever its size (16 rows of 1152 bytes: 11 bytes a clock, half of what HBM delivers), so a stage is fetched whole or in
// copies of a row's 1.7 KB and more where that fits.  Measured against the kernel before (eight warps to a tile with a barrier
// per tile, fragments of half a super-block; one-column arithmetic in launches of four columns for IQ2 / IQ1 / Q2_K and per-32
// columns): seven columns, 2 x 17408 x 5120 IQ3_XXS 41.8 -> 37.2 us, 65536 x 5120 Q6_K 78.5 -> 70.6; two columns, 2 x 17408 x
// 5120 Q4_K 27.9 -> 22.0; four columns, 2 x 17408 x 5120 IQ2_XS 46.9 -> 37.0, IQ1_S 45.1 -> 30.3, 5120 x 17408 Q2_K 34.1 -> 26.4;
// the 7-column pass 7.04 -> 6.38 ms (6.11 with the divisions as they are rated now), the four-column pass on 2- and 3-bit blocks 697 -> 588 us.
// Every column is computed by the same instructions whatever nb is, so column c of an nb-column call is
// bit-identical to a 1-column call on that column (the reference promises the same: src/cuda/gemv.cuh:31-34).
//
// A32: the columns come in the reference GPU path's per-32 format (int8 values, one scale per 32).  The formats that the
// one-column kernel serves with Q8_K blocks (IQ2_*, IQ1_*, Q2_K) and all per-32 columns give the one-column launch's bits: the
// same integer sums, the same float products, added in the order of its lane reduction (the sub-blocks of a super-block
// pairwise, then the super-blocks of a slice pairwise, then the slices in order), never in K-parts.
#pragma once
#include "q38b_act.cuh"
#include "q38b_decode1n.cuh"
#include "q38b_pipe.cuh"

namespace q38b {

constexpr int TILE_ROWS = 16;
constexpr int GEMV_MAX_WARPS = 20;  // consumer warps at most: with the producer and the adding warp 22, which leave a thread 80 registers
constexpr int GEMV_MAX_STAGES = 24;
constexpr int GEMV_TILEBUF = 2;     // tiles whose sums a group of warps holds: written, being added
constexpr int GEMV_HEADER = 1664;   // barriers and flags in front of the staged activations

constexpr int GEMV_MAX_MATS = 3;
constexpr int GEMV_MAX_PARTS = 32;
constexpr uint32_t PART_EMPTY = 0xFFFFFFFFu;   // a slot of the K-part scratch area that holds no sums (the area rests in this state)

// Columns of staged activations lie this many bytes off a multiple of 128: the four (8-byte loads of a half warp) or eight
// (4-byte loads of the k16 formats) columns that meet in one load then fall on different banks.
__host__ __device__ constexpr int act_skew(int fmt) { return fmt == T_Q6_K || fmt == T_Q2_K ? 16 : 32; }
// bytes of staged activation sums per column and super-block (mins() of q38b_decode.cuh)
__host__ __device__ constexpr int bsum_bytes(int fmt, bool a32) { return a32 ? 0 : fmt == T_Q4_K || fmt == T_Q5_K ? 16 : fmt == T_Q2_K ? 32 : 0; }
__host__ __device__ constexpr bool sign_table(int fmt) { return fmt == T_IQ3_XXS || fmt == T_IQ2_XXS || fmt == T_IQ2_XS; }
// a run of zeros beside the activations (q_half of FragEnv)
__host__ __device__ constexpr bool wants_zeros(int fmt) { return fmt == T_IQ2_XS || fmt == T_IQ2_S || fmt == T_IQ1_M; }

struct GemvArgs {
    // up to three matrices of one format, K and row stride on the same activation columns: their 16-row tiles form one
    // sequence (matrix 0's, then matrix 1's, ...), one launch replaces three
    const uint8_t* W_more[GEMV_MAX_MATS - 1];
    float* y_more[GEMV_MAX_MATS - 1];
    long long y_ld_more[GEMV_MAX_MATS - 1];
    int M_more[GEMV_MAX_MATS - 1];
    int tile_start[GEMV_MAX_MATS];   // first tile of each matrix (unused ones = n_tiles)
    const uint8_t* W;        // [M] rows, row_bytes apart, GGUF blocks
    long long row_bytes;
    const uint8_t* xq;       // Q8_K blocks (A32: int8 values); column c starts xq_ld bytes after column c - 1; or nullptr:
    long long xq_ld;
    const float* x_f32;      // then the columns as floats (column c at x_f32 + c * x_f32_ld), quantized to Q8_K by every CTA in its prologue
    long long x_f32_ld;
    const float* xd32;       // A32: one scale per 32 values, xd32_ld floats between the columns
    long long xd32_ld;
    float* y;                // y[c * y_ld + r]
    long long y_ld;
    float* y_peer[7];        // the same output position in the other GPUs' buffers (peer stores), n_peers used
    float* y_peer_more[GEMV_MAX_MATS - 1][7];   // the same for the further matrices of the launch
    int n_peers;
    int static_weights;     // 1: W was written long before this launch, the producer need not wait for earlier kernels
    int* status;             // device status word (OR of ST_* bits)
    const uint32_t* codebook;   // device copy of the format's codebook or grid codes (or nullptr)
    int K, M, nb, accumulate;
    int nsb;                 // super-blocks per row
    int n_tiles;
    int item_sb;             // super-blocks of a work item, at most (whole rows: nsb; K-parts: the longest part's)
    int chunk_sb;            // super-blocks per stage (the last chunk of an item may be shorter)
    int unit_log2;           // a warp takes 1 << unit_log2 super-blocks in a row: 1, 2 or 4
    int kw, groups;          // warps that share a tile; groups of them that take tiles in turn
    int contiguous;          // 1: a stage is 16 whole packed rows, fetched by one bulk copy
    int n_parts;             // K-parts of a row (1: the whole row is one work item per tile)
    int part_sb0[GEMV_MAX_PARTS + 1];   // first super-block of each part; [n_parts] = nsb
    int act_sb;              // super-blocks of activations a CTA stages per column (nsb, or two parts' worth)
    float* parts;            // n_parts > 1: 128 sums (16 rows x 8 columns) per (tile, part); PART_EMPTY between launches
    int* part_count;         // ... and per tile how many parts are written (zero between launches)
    int n_stages;
    int cols;                // columns whose sums are kept: nb rounded up to even
    int slots;               // 16 x cols sums per tile (one per unit)
    int slot_stride;         // bytes between the rows inside a stage
    int stage_bytes;
    // shared-memory offsets (bytes)
    int off_actd, off_actq, off_bsum, off_zero, off_cb, off_sgn, off_red, off_stage;
};

// The value of a super-block (of a sub-block: A32, Q8_0) enters these sums in the order of the one-column kernel's lane
// reduction: pairs of sub-blocks, pairs of pairs, then pairs of super-blocks.
struct PairSums {
    float p0[4], p1[4], p2[4];
    __device__ __forceinline__ void sub(int s, const float (&f)[4], float (&sb)[4]) {   // s = 0..7 in turn; sb: the eight's sum after s = 7
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if ((s & 1) == 0) { p0[i] = f[i]; continue; }
            const float a = p0[i] + f[i];
            if ((s & 2) == 0) { p1[i] = a; continue; }
            const float b = p1[i] + a;
            if ((s & 4) == 0) { p2[i] = b; continue; }
            sb[i] = p2[i] + b;
        }
    }
};

template <int FMT, bool A32, bool PARTED>
__global__ void __launch_bounds__(32 * (2 + GEMV_MAX_WARPS), 1) gemv_kernel(const GemvArgs a) {
    using U = Unit<FMT>;
    constexpr int BB = U::BLOCK_BYTES;
    constexpr int NW = GEMV_MAX_WARPS;                      // warps that set up tables and activations; the first kw * groups consume
    static_assert(!(A32 && FMT == T_Q6_K), "per-32 columns of Q6_K run on the one-column kernel's arithmetic");
    extern __shared__ __align__(128) uint8_t smem_raw[];   // plain pointer arithmetic from here on keeps loads in the shared space
    uint8_t* smem = smem_raw;
    uint64_t* full = (uint64_t*)smem;                       // [GEMV_MAX_STAGES]
    uint64_t* empty = full + GEMV_MAX_STAGES;               // [GEMV_MAX_STAGES]
    uint64_t* tbar = empty + GEMV_MAX_STAGES;               // [groups][GEMV_TILEBUF] a tile's units have put their sums down
    uint64_t* tfree = tbar + GEMV_MAX_WARPS * GEMV_TILEBUF; // [groups][GEMV_TILEBUF] ... and they have been added up
    volatile int* abort_flag = (volatile int*)(tfree + GEMV_MAX_WARPS * GEMV_TILEBUF);
    static_assert(8 * (2 * GEMV_MAX_STAGES + 2 * GEMV_MAX_WARPS * GEMV_TILEBUF) + 8 <= GEMV_HEADER, "header");
    // Work items of this CTA, k = 0, 1, ...: whole rows: tile blockIdx.x + gridDim.x * k.  K-parts: the items (part, tile),
    // part-major, are cut into gridDim.x equal ranges.
    const long long n_items = (long long)a.n_tiles * (PARTED ? a.n_parts : 1);
    const long long item_lo = PARTED ? n_items * blockIdx.x / gridDim.x : 0;
    const int my_items = PARTED ? (int)(n_items * (blockIdx.x + 1) / gridDim.x - item_lo)
                                : (a.n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // (the grid is never larger than n_tiles)
    // the activations this CTA stages: super-blocks [win0, win0 + win_sb) of every column
    const int part_first = PARTED ? (int)(item_lo / a.n_tiles) : 0;
    const int part_last = PARTED && my_items > 0 ? (int)((item_lo + my_items - 1) / a.n_tiles) : part_first;
    const int win0 = PARTED ? a.part_sb0[part_first] : 0;
    const int win_sb = PARTED ? a.part_sb0[part_last + 1] - win0 : a.nsb;
    const int act_ld = a.act_sb * 256 + act_skew(FMT);      // bytes between the staged columns
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (warp == 0) {
        if (lane == 0) *abort_flag = 0;
        for (int i = lane; i < a.n_stages; i += 32) {
            mbar_init(smem_u32(&full[i]), TILE_ROWS);         // one arrival per row copy
            mbar_init(smem_u32(&empty[i]), a.kw);             // one per warp that reads the stage
        }
        for (int i = lane; i < a.groups * GEMV_TILEBUF; i += 32) {
            mbar_init(smem_u32(&tbar[i]), a.kw);
            mbar_init(smem_u32(&tfree[i]), 1);
        }
        mbar_fence_init();
    }
    __syncthreads();
    pdl_launch_dependents();

    const int packed_row = a.nsb * BB;
    // The walk over this CTA's items (nothing is divided on the way).
    struct Walk { int k, part, gtile, sb0, nsb; } w;
    w.k = 0;
    w.part = part_first;
    w.gtile = PARTED ? (int)(item_lo - (long long)part_first * a.n_tiles) : (int)blockIdx.x;
    w.sb0 = PARTED ? a.part_sb0[part_first] : 0;
    w.nsb = PARTED ? a.part_sb0[part_first + 1] - w.sb0 : a.nsb;
    auto next_item = [&](Walk& w) {
        w.k++;
        if (PARTED) {
            if (++w.gtile == a.n_tiles) {
                w.gtile = 0;
                w.part++;
                if (w.part < a.n_parts) { w.sb0 = a.part_sb0[w.part]; w.nsb = a.part_sb0[w.part + 1] - w.sb0; }
            }
        } else {
            w.gtile += (int)gridDim.x;
        }
    };

    if (warp == 0) {
        // ---------------- producer: resident weights do not depend on earlier kernels, start at once ----------------
        if (!a.static_weights) pdl_wait_prior();   // otherwise W may be the output of the kernel before this one
        if (lane < TILE_ROWS) {
            const int r = lane;                        // this lane's row of a tile
            int stage = 0;
            uint32_t use = 0;
            for (; w.k < my_items; next_item(w)) {
                const int mi = (w.gtile >= a.tile_start[1]) + (w.gtile >= a.tile_start[2]);
                const int row0 = (w.gtile - a.tile_start[mi]) * TILE_ROWS;
                const uint8_t* Wm = mi == 0 ? a.W : a.W_more[mi - 1];
                const int Mm = mi == 0 ? a.M : a.M_more[mi - 1];
                const int rows_here = min(TILE_ROWS, Mm - row0);
                const uintptr_t safe_end = ((uintptr_t)Wm + (uintptr_t)(Mm - 1) * a.row_bytes + packed_row) & ~(uintptr_t)15;
                for (int c0 = 0; c0 < w.nsb; c0 += a.chunk_sb) {
                    const uint32_t fb = smem_u32(&full[stage]);
                    mbar_wait_bounded(smem_u32(&empty[stage]), use ^ 1u, abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT);
                    uint8_t* slot = smem + a.off_stage + (size_t)stage * a.stage_bytes;
                    uintptr_t src = 0;
                    long long len = 0;
                    if (a.contiguous) {
                        if (r == 0) {
                            src = (uintptr_t)Wm + (uintptr_t)row0 * a.row_bytes;
                            len = (long long)rows_here * a.row_bytes;
                        }
                    } else if (r < rows_here) {
                        const int off = (w.sb0 + c0) * BB;
                        src = (uintptr_t)Wm + (uintptr_t)(row0 + r) * a.row_bytes + (uintptr_t)off;
                        len = min(a.chunk_sb, w.nsb - c0) * BB;
                        slot += (size_t)r * a.slot_stride;
                    }
                    if (len <= 0) {
                        mbar_arrive(fb);
                    } else {
                        const uintptr_t lo = src & ~(uintptr_t)15;
                        uintptr_t hi = (src + len + 15) & ~(uintptr_t)15;
                        if (hi > safe_end) {
                            // the last bytes of the tensor do not fill a 16-byte unit: fetch them with plain loads
                            hi = safe_end > lo ? safe_end : lo;
                            for (uintptr_t p = hi; p < src + len; p += 2)
                                if (p >= src) *(uint16_t*)(slot + (p - lo)) = *(const uint16_t*)p;
                        }
                        const uint32_t bytes = (uint32_t)(hi - lo);
                        if (bytes) {
                            mbar_arrive_expect_tx(fb, bytes);
                            bulk_copy_g2s(smem_u32(slot), (const void*)lo, bytes, fb);
                        } else {
                            mbar_arrive(fb);
                        }
                    }
                    if (++stage == a.n_stages) { stage = 0; use ^= 1u; }
                }
            }
        }
        return;
    }

    const int g = lane >> 2, t = lane & 3;
    float* red = (float*)(smem + a.off_red);         // [groups][GEMV_TILEBUF][slots][16 rows][cols]
    const int slot_sums = 16 * a.cols;
    const bool keeps = 2 * t < a.cols;
    if (warp == 1 + NW) {
        // ---------------- the warp that adds up tiles ----------------
        pdl_wait_prior();                            // y may still be read by earlier kernels
        // K-parts: adds up the parts of tile ft (this warp counted the last one) and stores the rows
        auto add_up = [&](int ft) {
            const int mi = (ft >= a.tile_start[1]) + (ft >= a.tile_start[2]);
            const int tile = ft - a.tile_start[mi];
            const int Mm = mi == 0 ? a.M : a.M_more[mi - 1];
            const long long ld = mi == 0 ? a.y_ld : a.y_ld_more[mi - 1];
            float* ym = mi == 0 ? a.y : a.y_more[mi - 1];
            float* sp = a.parts + (size_t)ft * a.n_parts * 128 + lane;
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            const long long t0 = clock64();
            for (int p0 = 0; p0 < a.n_parts; p0 += 4) {   // the loads of four parts go out together
                uint32_t u[4][4];
                bool all = false;
                while (!all) {
                    all = true;
#pragma unroll
                    for (int pp = 0; pp < 4; pp++)
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            u[pp][i] = 0u;
                            if (p0 + pp < a.n_parts)
                                asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(u[pp][i]) : "l"(sp + (p0 + pp) * 128 + 32 * i) : "memory");
                        }
#pragma unroll
                    for (int pp = 0; pp < 4; pp++)
#pragma unroll
                        for (int i = 0; i < 4; i++) all = all && u[pp][i] != PART_EMPTY;
                    all = __all_sync(0xffffffffu, all);
                    if (!all && clock64() - t0 > WAIT_BUDGET_CYCLES) {
                        if (lane == 0) atomicOr(a.status, ST_WAIT_FULL_TIMEOUT);
                        break;
                    }
                }
#pragma unroll
                for (int pp = 0; pp < 4; pp++)
                    if (p0 + pp < a.n_parts) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            v[i] = p0 + pp == 0 ? __uint_as_float(u[pp][i]) : v[i] + __uint_as_float(u[pp][i]);
                            __stcg((uint32_t*)(sp + (p0 + pp) * 128 + 32 * i), PART_EMPTY);
                        }
                    }
            }
            if (lane == 0) a.part_count[ft] = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = tile * TILE_ROWS + g + 8 * (i >> 1);
                const int col = 2 * t + (i & 1);
                if (row < Mm && col < a.nb) {
                    float* yo = ym + (size_t)col * ld + row;
                    const float out = a.accumulate ? *yo + v[i] : v[i];
                    *yo = out;
                    for (int pr = 0; pr < a.n_peers; pr++) (mi == 0 ? a.y_peer[pr] : a.y_peer_more[mi - 1][pr])[(size_t)col * ld + row] = out;
                }
            }
        };
        int pending = -1, pending_tile = -1;             // K-parts: the count drawn for the last part this warp put down (lane 0), and its tile

        // Adds up the tile in buffer `at` (its units have arrived: `par`) and stores it or, K-parts, puts it into the scratch area.
        // Units of one super-block: pairs, pairs of pairs, then the slices of four in order; of two: pairs; of four: in order.
        auto finish = [&](const Walk& f, int at, uint32_t par) {
            mbar_wait_bounded(smem_u32(&tbar[at]), par, abort_flag, a.status, ST_WAIT_FULL_TIMEOUT);
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (keeps) {
                const float* r0 = red + (size_t)at * a.slots * slot_sums + g * a.cols + 2 * t;
                const int n = (f.nsb + (1 << a.unit_log2) - 1) >> a.unit_log2;
                auto slot = [&](int u, float (&x)[4]) {
                    float2 lo = make_float2(0.f, 0.f), hi = lo;
                    if (u < n) {
                        lo = *(const float2*)(r0 + u * slot_sums);
                        hi = *(const float2*)(r0 + u * slot_sums + 8 * a.cols);
                    }
                    x[0] = lo.x; x[1] = lo.y; x[2] = hi.x; x[3] = hi.y;
                };
                const int per = 4 >> a.unit_log2;                // units of a slice
                for (int u = 0; u < n; u += per) {
                    float x0[4], x1[4], x2[4], x3[4];
                    slot(u, x0);
                    if (per > 1) slot(u + 1, x1);
                    if (per > 2) { slot(u + 2, x2); slot(u + 3, x3); }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (per > 1) x0[i] += x1[i];
                        if (per > 2) x0[i] += x2[i] + x3[i];
                        v[i] += x0[i];
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tfree[at]));
            if (PARTED) {   // the tile's other parts may be other CTAs' work: put the sums down, count, look at the count with the next item
#pragma unroll
                for (int i = 0; i < 4; i++) __stcg(a.parts + ((size_t)f.gtile * a.n_parts + f.part) * 128 + 32 * i + lane, v[i]);
                __syncwarp();
                const int before = pending, before_tile = pending_tile;
                if (lane == 0) pending = atomicAdd(a.part_count + f.gtile, 1);
                pending_tile = f.gtile;
                if (before_tile >= 0 && __shfl_sync(0xffffffffu, before, 0) == a.n_parts - 1) add_up(before_tile);
                return;
            }
            const int mi = (f.gtile >= a.tile_start[1]) + (f.gtile >= a.tile_start[2]);
            const int tile = f.gtile - a.tile_start[mi];
            const int Mm = mi == 0 ? a.M : a.M_more[mi - 1];
            const long long ld = mi == 0 ? a.y_ld : a.y_ld_more[mi - 1];
            float* ym = mi == 0 ? a.y : a.y_more[mi - 1];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = tile * TILE_ROWS + g + 8 * (i >> 1), col = 2 * t + (i & 1);
                if (row < Mm && col < a.nb) {
                    float* yo = ym + (size_t)col * ld + row;
                    const float out = a.accumulate ? *yo + v[i] : v[i];
                    *yo = out;
                    for (int pr = 0; pr < a.n_peers; pr++) (mi == 0 ? a.y_peer[pr] : a.y_peer_more[mi - 1][pr])[(size_t)col * ld + row] = out;
                }
            }
        };

        int grp = 0, buf = 0;
        uint32_t par = 0;
        for (; w.k < my_items; next_item(w)) {       // the items in order: group k % groups, its buffers in turn
            finish(w, grp * GEMV_TILEBUF + buf, par);
            if (++grp == a.groups) {
                grp = 0;
                if (++buf == GEMV_TILEBUF) { buf = 0; par ^= 1u; }
            }
        }
        if (PARTED && pending_tile >= 0 && __shfl_sync(0xffffffffu, pending, 0) == a.n_parts - 1) add_up(pending_tile);
        return;
    }

    // ---------------- consumers ----------------
    const int cw = warp - 1, ctid = tid - 32;
    float* actd = (float*)(smem + a.off_actd);       // [win_sb][8] scales (A32: [8 win_sb][8])
    uint8_t* actq = smem + a.off_actq;               // [nb][act_ld], staged order
    uint32_t* cbw = (uint32_t*)(smem + a.off_cb);
    if constexpr (U::CODEBOOK_ENTRIES > 0) {
        constexpr int REP_LOG2 = cb1_rep_log2(FMT), WORDS = U::CODEBOOK_ENTRIES << REP_LOG2;
#pragma unroll 4
        for (int i = ctid; i < WORDS / 4; i += NW * 32) {
            const uint32_t v = a.codebook[i >> (REP_LOG2 - 2)];
            ((uint4*)cbw)[i] = make_uint4(v, v, v, v);
        }
    } else if constexpr (gridx_copies(FMT) > 0) {
        // two copies of an entry are 16 bytes: a warp's stores cover 512 consecutive bytes
        constexpr int PAIRS = gridx_copies(FMT) / 2;
#pragma unroll 4
        for (int i = ctid; i < code16_entries(FMT) * PAIRS; i += NW * 32) {
            uint32_t lo, hi;
            gridx_entry<FMT>(((const uint16_t*)a.codebook)[i / PAIRS], lo, hi);
            if (FMT == T_IQ1_S || FMT == T_IQ1_M) {   // eight times the level -1, 0, 1 as signed bytes
                lo = ((lo | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
                hi = ((hi | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
            }
            ((uint4*)cbw)[i] = make_uint4(lo, hi, lo, hi);
        }
    }
    if constexpr (sign_table(FMT)) {
        uint2* sg = (uint2*)(smem + a.off_sgn);
#pragma unroll 1
        for (int i = ctid; i < 128 * SIGN_COPIES; i += NW * 32) {
            uint32_t lo, hi;
            sign_masks7((uint32_t)i / SIGN_COPIES, lo, hi);
            sg[i] = make_uint2(lo, hi);
        }
    }
    if (wants_zeros(FMT))
        for (int i = ctid; i < 66; i += NW * 32) ((uint32_t*)(smem + a.off_zero))[i] = 0u;
    pdl_wait_prior();   // activations come from the previous kernel of the stream
    // blocks (column c, super-block sb of the window) go round the warps; stepped, not divided
    struct Block { int c, sb; };
    auto step = [&](Block& b, int n) {
        b.sb += n;
        while (b.sb >= win_sb) { b.sb -= win_sb; b.c++; }
    };
    Block at = {0, 0};
    step(at, cw);
    // Sums of a block's activations, as digits (mins() of q38b_decode.cuh).  Floats: a lane has eight values in a row (w0, w1); blocks: words
    // l % 4 and l % 4 + 4 of 32.  Either way four lanes have a sub-block; sixteen values are two of them or one word of each.
    constexpr int BS = bsum_bytes(FMT, A32);
    const bool floats = !A32 && a.x_f32;
    auto put_bsum = [&](int c, int sb, uint32_t w0, uint32_t w1) {
        if constexpr (BS > 0) {
            uint8_t* to = smem + a.off_bsum + (sb * 8 + c) * BS;
            const int s0 = __dp4a((int)w0, 0x01010101, 0), s1 = __dp4a((int)w1, 0x01010101, 0);
            if constexpr (FMT == T_Q2_K) {
                int x = floats ? s0 + s1 : s0, y = s1;
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                if (floats) {
                    if ((lane & 1) == 0) { to[lane >> 1] = (uint8_t)(x & 63); to[16 + (lane >> 1)] = (uint8_t)(x >> 6); }
                } else {
                    x += __shfl_xor_sync(0xffffffffu, x, 2);
                    y += __shfl_xor_sync(0xffffffffu, y, 1);
                    y += __shfl_xor_sync(0xffffffffu, y, 2);
                    if ((lane & 3) == 0) {
                        to[lane >> 1] = (uint8_t)(x & 63); to[16 + (lane >> 1)] = (uint8_t)(x >> 6);
                        to[(lane >> 1) + 1] = (uint8_t)(y & 63); to[17 + (lane >> 1)] = (uint8_t)(y >> 6);
                    }
                }
            } else {
                int x = s0 + s1;
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                x += __shfl_xor_sync(0xffffffffu, x, 2);
                if ((lane & 3) == 0) { to[lane >> 2] = (uint8_t)(x & 63); to[8 + (lane >> 2)] = (uint8_t)(x >> 6); }
            }
        }
    };
    constexpr int DPB = A32 ? 64 : 8;                // staged scale slots per super-block
    for (int i = ctid; i < win_sb * DPB; i += NW * 32)
        if ((i & 7) >= a.nb) actd[i] = 0.0f;
    if (!A32 && a.x_f32) {
        // quantize the columns here (every CTA, the arithmetic of quantize_q8k_kernel): a warp takes two blocks of
        // 256 values at a time, their loads going out together (four: the code no longer fits what the SM has at hand)
        constexpr int QB = 2;
#pragma unroll 1
        while (at.c < a.nb) {
            float v[QB][8], d[QB];
            uint32_t w0[QB], w1[QB];
            Block blk[QB];
#pragma unroll
            for (int j = 0; j < QB; j++) {
                blk[j] = at;
                const float* src = a.x_f32 + (size_t)min(at.c, a.nb - 1) * a.x_f32_ld + (size_t)(win0 + at.sb) * 256 + 8 * lane;
                const float4 lo = *(const float4*)src, hi = *(const float4*)(src + 4);
                v[j][0] = lo.x; v[j][1] = lo.y; v[j][2] = lo.z; v[j][3] = lo.w;
                v[j][4] = hi.x; v[j][5] = hi.y; v[j][6] = hi.z; v[j][7] = hi.w;
                step(at, NW);
            }
            q8k_blocks_core<QB>(v, w0, w1, d);
#pragma unroll
            for (int j = 0; j < QB; j++) {
                const int c = blk[j].c, sb = blk[j].sb;
                if (c >= a.nb) break;
                if (lane == 0) actd[sb * 8 + c] = d[j];
                uint8_t* dst = actq + (size_t)c * act_ld + sb * 256;
                if (FMT == T_IQ4_XS) {
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const int k = 8 * lane + e;
                        dst[(k & ~31) + act_stage_pos(FMT, k & 31)] = (uint8_t)((e < 4 ? w0[j] : w1[j]) >> (8 * (e & 3)));
                    }
                } else {
                    *(uint2*)(dst + 8 * lane) = make_uint2(w0[j], w1[j]);
                }
                put_bsum(c, sb, w0[j], w1[j]);
            }
        }
    } else {
        // copy the blocks' scales and values: one warp per 256 values (64 words: lane l takes words w and
        // w + 4 of the 32-value group l / 4, w = l % 4), the loads of four blocks going out together
        constexpr int SB = 4;
        const int wofs = 8 * (lane >> 2) + (lane & 3);
#pragma unroll 1
        while (at.c < a.nb) {
            uint32_t w0[SB], w1[SB], dw[SB];
            Block dst_at[SB];
#pragma unroll
            for (int jb = 0; jb < SB; jb++) {
                dst_at[jb] = at;
                w0[jb] = w1[jb] = dw[jb] = 0u;
                if (at.c < a.nb) {
                    const int c = at.c, sb = win0 + at.sb;
                    const uint32_t* blk = (const uint32_t*)(a.xq + (size_t)c * a.xq_ld + (A32 ? (size_t)sb * 256 : (size_t)sb * Q8K_BYTES + 4));
                    w0[jb] = blk[wofs];
                    w1[jb] = blk[4 + wofs];
                    if (A32) {
                        if (lane < 8) dw[jb] = __float_as_uint(a.xd32[(size_t)c * a.xd32_ld + (size_t)sb * 8 + lane]);
                    } else if (lane == 0) {
                        dw[jb] = blk[-1];
                    }
                }
                step(at, NW);
            }
#pragma unroll
            for (int jb = 0; jb < SB; jb++) {
                const int c = dst_at[jb].c, sb = dst_at[jb].sb;
                if (c >= a.nb) break;
                if (lane < (A32 ? 8 : 1)) actd[sb * DPB + 8 * lane + c] = __uint_as_float(dw[jb]);
                uint8_t* dst = actq + (size_t)c * act_ld + sb * 256 + 32 * (lane >> 2);
                if (FMT == T_IQ4_XS) {
                    // act_stage_pos: value k of the group goes to 8 (k % 16 / 4) + 2 (k % 4) + k / 16, i.e. the bytes of
                    // words w and w + 4 interleaved
                    *(uint2*)(dst + 8 * (lane & 3)) = make_uint2(prmt(w0[jb], w1[jb], 0x5140u), prmt(w0[jb], w1[jb], 0x7362u));
                } else {
                    *(uint32_t*)(dst + 4 * (lane & 3)) = w0[jb];
                    *(uint32_t*)(dst + 16 + 4 * (lane & 3)) = w1[jb];
                }
                put_bsum(c, sb, w0[jb], w1[jb]);
            }
        }
    }
    named_bar_sync(15, NW * 32);
    if (cw >= a.kw * a.groups) return;

    FragEnv env;
    env.t = t;
    if constexpr (gridx_copies(FMT) > 0) {
        env.cb_shift = gridx_copies(FMT) == 16 ? 7 : gridx_copies(FMT) == 8 ? 6 : 5;
        env.cb = sp_from(cbw) + 8 * (lane & (gridx_copies(FMT) - 1));
    } else {
        env.cb_shift = cb1_rep_log2(FMT) + 2;
        env.cb = sp_from(cbw) + 4 * (lane & ((1 << cb1_rep_log2(FMT)) - 1));
    }
    env.sgn = sp_from(smem + a.off_sgn) + 8 * (lane & (SIGN_COPIES - 1));
    const SP bsum0 = sp_from(smem + a.off_bsum) + (g * BS + 4 * t - win0 * 8 * BS);
    const SP zero = sp_from(smem + a.off_zero);
    const SP q_col = sp_from(actq) + ((g < a.nb ? g : 0) * act_ld + U::ACT_STEP * t - win0 * 256);   // indexed by the super-block's number in the row
    const SP d_col = sp_from(actd) + (8 * t - win0 * DPB * 4);
    const SP stage0 = sp_from(smem + a.off_stage);
    const uint32_t rb32 = (uint32_t)a.row_bytes;
    const uint32_t rb_step = a.contiguous ? 0u : 8u * rb32;   // rows of a contiguous stage share the copy's low address bits
    const uint32_t rb_g = a.contiguous ? 0u : (uint32_t)g * rb32;

    const int grp = cw / a.kw, uw = cw - grp * a.kw; // group, and this warp's place in it
    uint64_t* my_tbar = tbar + grp * GEMV_TILEBUF;
    uint64_t* my_tfree = tfree + grp * GEMV_TILEBUF;
    float* my_red = red + (size_t)grp * GEMV_TILEBUF * a.slots * slot_sums + g * a.cols + 2 * t;

    // This group's items: grp, grp + groups, ...  (several groups: one chunk an item and a multiple of `groups` stages, so that
    // a group meets every use of its stages)
    for (int i = 0; i < grp; i++) next_item(w);
    int stage = grp, buf = 0;
    uint32_t stage_par = 0, buf_par = 0;
    while (w.k < my_items) {
        const int mi = (w.gtile >= a.tile_start[1]) + (w.gtile >= a.tile_start[2]);
        const int tile = w.gtile - a.tile_start[mi];
        const uint32_t tile_lo = (uint32_t)(uintptr_t)(mi == 0 ? a.W : a.W_more[mi - 1]) + (uint32_t)(tile * TILE_ROWS) * rb32;
        // before this warp's first sums of the tile, and before it arrives: the tile before in this buffer has been added up
        bool taken = false;
        auto take_buffer = [&]() {
            if (!taken) mbar_wait_bounded(smem_u32(&my_tfree[buf]), buf_par ^ 1u, abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT);
            taken = true;
        };
        for (int c0 = 0; c0 < w.nsb; c0 += a.chunk_sb) {
            mbar_wait_bounded(smem_u32(&full[stage]), stage_par, abort_flag, a.status, ST_WAIT_FULL_TIMEOUT);
            // low address bits of row 0 of the tile at this stage's first byte (a copy keeps its low 4 address bits)
            const uint32_t src_lo = tile_lo + (a.contiguous ? 0u : (uint32_t)((w.sb0 + c0) * BB));
            const SP st = stage0 + (stage * a.stage_bytes + g * a.slot_stride);
            const SP rowA = st + (int)((src_lo + rb_g) & 15u);
            const SP rowB = st + (8 * a.slot_stride + (int)((src_lo + rb_g + rb_step) & 15u));
            const int chunk_end = min(a.chunk_sb, w.nsb - c0);
        for (int u0 = uw << a.unit_log2; u0 < chunk_end; u0 += a.kw << a.unit_log2) {
        const int n_sb = min(1 << a.unit_log2, chunk_end - u0), sb0 = w.sb0 + c0 + u0;
        SP pA = rowA + u0 * BB, pB = rowB + u0 * BB;
        float acc[4] = {0.f, 0.f, 0.f, 0.f}, first[4] = {0.f, 0.f, 0.f, 0.f};   // sums of super-blocks 2, 3 (0, 1 while it is at those) and 0, 1
#pragma unroll 1
        for (int b = 0; b < n_sb; b++, pA = pA + BB, pB = pB + BB) {
            env.q = q_col + (sb0 + b) * 256;
            if (wants_zeros(FMT)) {
                env.q_half[0] = t < 2 ? env.q : zero;
                env.q_half[1] = t < 2 ? zero : env.q;
            }
            const SP dq = d_col + (sb0 + b) * (DPB * 4);
            typename U::Row A, B;
            U::row(pA, t, A);
            U::row(pB, t, B);
            int cm[4] = {0, 0, 0, 0};
            float dA, mA, dB, mB, f[4];
            U::dd(pA, A, dA, mA);
            U::dd(pB, B, dB, mB);
            if constexpr (A32 || U::SCALE32) {
                PairSums ps;
                float dx0 = sp_ldf(dq), dx1 = sp_ldf(dq, 4);
                constexpr bool QPAIR = FMT == T_Q4_K || FMT == T_Q5_K;   // a lane of the one-column kernel owns a pair of sub-blocks there
                float kv[4], km[4];
#pragma unroll
                for (int h = 0; h < 2; h++)
                    U::template half<!U::HAS_MIN>(A, B, pA, pB, h, env, cm, [&](int s, const int (&v)[4]) {
                        if (A32) { dx0 = sp_ldf(dq, 32 * s); dx1 = sp_ldf(dq, 32 * s + 4); }
                        float x[4];
                        if constexpr (QPAIR) {
                            // d (dx0 sc0 lo + dx1 sc1 hi) - dmin (dx0 mn0 sum0 + dx1 mn1 sum1), as GranQ45K
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const float dx = (i & 1) ? dx1 : dx0;
                                if ((s & 1) == 0) {
                                    kv[i] = fmul_once(dx, (float)v[i]);
                                    km[i] = fmul_once(dx, (float)cm[i]);
                                } else {
                                    kv[i] = fmaf(dx, (float)v[i], kv[i]);
                                    km[i] = fmaf(dx, (float)cm[i], km[i]);
                                    x[i] = fmaf(-(i < 2 ? mA : mB), km[i], fmul_once(i < 2 ? dA : dB, kv[i]));
                                }
                                cm[i] = 0;
                            }
                            if (s & 1) {   // four pairs of sub-blocks a super-block
#pragma unroll
                                for (int i = 0; i < 4; i++) {
                                    if (((s >> 1) & 1) == 0) { ps.p0[i] = x[i]; continue; }
                                    const float two = ps.p0[i] + x[i];
                                    if (((s >> 1) & 2) == 0) ps.p1[i] = two;
                                    else f[i] = ps.p1[i] + two;
                                }
                            }
                        } else {
                            const float eA = U::SCALE32 ? U::d32(pA, s) : dA, eB = U::SCALE32 ? U::d32(pB, s) : dB;
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const float dx = (i & 1) ? dx1 : dx0, e = i < 2 ? eA : eB;
                                if (U::HAS_MIN) {
                                    x[i] = block_value_min(e * dx, v[i], (i < 2 ? mA : mB) * dx, cm[i]);
                                    cm[i] = 0;
                                } else {
                                    x[i] = block_value(e * dx * U::FACTOR, v[i]);
                                }
                            }
                            ps.sub(s, x, f);
                        }
                    });
            } else {
                int sumi[4] = {0, 0, 0, 0};
                if constexpr (BS > 0) {
                    env.bsum = bsum0 + (sb0 + b) * (8 * BS);
                    U::mins(A, B, env, cm);
                }
#pragma unroll
                for (int h = 0; h < 2; h++)
                    U::template half<true>(A, B, pA, pB, h, env, cm, [&](int, const int (&v)[4]) {
#pragma unroll
                        for (int i = 0; i < 4; i++) sumi[i] += v[i];
                    });
                const float dx0 = sp_ldf(dq), dx1 = sp_ldf(dq, 4);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float dx = (i & 1) ? dx1 : dx0, d = i < 2 ? dA : dB;
                    f[i] = U::HAS_MIN ? block_value_min(d * dx, sumi[i], (i < 2 ? mA : mB) * dx, cm[i]) : block_value(d * dx * U::FACTOR, sumi[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (b == 2) { first[i] = acc[i]; acc[i] = 0.0f; }
                acc[i] += f[i];
            }
        }
        take_buffer();
        if (keeps) {
            float* rt = my_red + (size_t)(buf * a.slots + ((c0 + u0) >> a.unit_log2)) * slot_sums;
            *(float2*)rt = make_float2(first[0] + acc[0], first[1] + acc[1]);
            *(float2*)(rt + 8 * a.cols) = make_float2(first[2] + acc[2], first[3] + acc[3]);
        }
        }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&empty[stage]));
            stage += a.groups;
            if (stage >= a.n_stages) { stage -= a.n_stages; stage_par ^= 1u; }
        }
        take_buffer();
        if (lane == 0) mbar_arrive(smem_u32(&my_tbar[buf]));
        if (++buf == GEMV_TILEBUF) { buf = 0; buf_par ^= 1u; }
        if (PARTED) {
            for (int i = 0; i < a.groups; i++) next_item(w);
        } else {
            w.k += a.groups;
            w.gtile += a.groups * (int)gridDim.x;
        }
    }
}

}  // namespace q38b
