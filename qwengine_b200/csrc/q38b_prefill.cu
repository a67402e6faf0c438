// q38b_prefill.cu -- dequant-on-the-fly prefill GEMM on the 5th-generation tensor cores (tcgen05 + TMEM).
//
//   Y[t][r] (+)= sum_k X[t][k] * W[r][k]      X bf16 [B][ldx], W GGUF blocks [M rows], Y fp32 [B][ldy]
//
// Replaces dequant_rows_f16 + gemm_f16 (cuBLAS) of the reference (src/cuda/prefill.cu:30-85, 802-851) by one kernel:
// the weights never exist dequantized in global memory.  One CTA owns a 128-row weight tile and up to 512 tokens:
//   * warps 0-15 fetch the rows' raw blocks one super-block ahead (whole 16-byte units into registers, then shared memory), a
//     lane expands one 32-weight sub-block with word operations (q38b_expand.cuh) into operand A: for token tiles over 256
//     K-major with the 128-byte swizzle in shared memory (a warp owns eight rows), for tiles of at most 256 in tensor memory
//     (a lane is a row);
//   * one thread streams the matching activation tiles (operand B, [tokens x 64] per K-slab) with tiled TMA loads
//     (hardware swizzle, zero fill past the last token; no multicast);
//   * one thread issues tcgen05.mma (kind::f16, M = 128, N = 16..256, K = 16; tiles over 256 tokens whose K is not shared: two
//     CTAs as a pair, M = 256) into one or two fp32
//     accumulators in tensor memory and commits each stage to its "empty" mbarrier;
//   * all 16 decode warps read the accumulators back (tcgen05.ld 32x32b) and store Y, 32 consecutive rows per warp and token.
// Where row tiles and token tiles alone leave SMs idle, the CTAs of a cluster share a tile's K: each multiplies a range
// of super-blocks and the partial sums meet through distributed shared memory, added in rank order.
// Measured on B200, 17408 x 5120 IQ3_XXS / 5120 x 17408 IQ4_XS with 1024 tokens: 211 / 286 us -> 161 / 194 us; in pairs 143
// for the former; 77 tokens of a whole Q4_K / Q6_K layer 698 -> 199 us, 154 us with operand A in tensor memory.  In tiles of at most 256 tokens
// the expanders set the pace, in tiles of 500 the tensor core and the shared-memory traffic do.
// All mbarrier waits are bounded; tensor memory is released before the kernel returns, also after a timeout.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "../../include/q38b200.h"
#include "q38b_expand.cuh"
#include "q38b_internal.h"
#include "q38b_pipe.cuh"

using namespace q38b;

namespace {

constexpr int PF_ROWS = 128;       // weight rows per CTA (MMA M)
constexpr int PF_MAX_N = 256;      // tokens per accumulator (MMA N), at most
constexpr int PF_KSLAB = 64;       // K elements per activation stage: one 128-byte swizzle row of bf16
// The two operands have rings of their own: dequantized weights two deep in stages of half a super-block (two K-slabs,
// 32 KB), activation tiles of one slab and one accumulator as deep as fits (four of 256 tokens, up to eight of fewer).
constexpr int PF_A_STAGES = 2, PF_B_MAX_STAGES = 8;
constexpr int PF_A_SLAB_BYTES = PF_ROWS * PF_KSLAB * 2;   // 16 KB
constexpr int PF_A_BYTES = 2 * PF_A_SLAB_BYTES;
constexpr int PF_DECODE_WARPS = 16, PF_WARP_ROWS = PF_ROWS / PF_DECODE_WARPS;
constexpr int PF_THREADS = 32 * (PF_DECODE_WARPS + 2);    // + TMA warp + MMA warp
constexpr int PF_MAX_SPLITS = 8;   // CTAs that share a tile's K (portable cluster size)

// Raw bytes a warp keeps of each of its rows: a super-block (Q8_0, whose halves are self-contained, half of one), at the
// low four bits of its global address, read in whole 16-byte pieces.  The distance between rows is an odd number of
// pieces, so that the eight rows a load instruction touches start on different banks.
__host__ __device__ constexpr int pf_raw_bytes(int fmt) { return fmt == T_Q8_0 ? 136 : block_bytes(fmt); }
__host__ __device__ constexpr int pf_pieces(int fmt) { return (pf_raw_bytes(fmt) + 14 + 15) / 16; }
__host__ __device__ constexpr int pf_pitch(int fmt) { return 16 * (pf_pieces(fmt) | 1); }
__host__ __device__ constexpr int pf_raw_smem(int fmt) { return PF_ROWS * pf_pitch(fmt) + 16; }   // + what the last row's word loads read past its end
// Operand A in tensor memory (one accumulator, a tile of up to 256 tokens): a decode warp's lanes are 32 rows, an odd number of the
// format's loads (16, 8 or 4 bytes) apart; two buffers, as four warps share a quarter of the rows.
__host__ __device__ constexpr int pf_pitch_ta(int fmt, bool aligned) {
    return aligned && (fmt == T_Q4_K || fmt == T_Q5_K) ? pf_pitch(fmt) : 16 * pf_pieces(fmt) + (aligned && fmt == T_IQ4_XS ? 8 : 4);
}
__host__ __device__ constexpr int pf_raw_ta(int fmt) { return (PF_ROWS * 16 * (pf_pieces(fmt) + 1) + 16 + 127) / 128 * 128; }   // one buffer, any pitch
__host__ __device__ constexpr int pf_fixed_smem(int fmt, bool ta) {
    return 1024 + (ta ? 2 * pf_raw_ta(fmt) : PF_A_STAGES * PF_A_BYTES + pf_raw_smem(fmt)) + grid_table_bytes(fmt) + 16;
}
constexpr int PF_TA_STAGE_COLS = 64;   // 128 rows x 128 K of 16-bit weights: 64 columns of tensor memory
constexpr int PF_TA_MAX_STAGES = 6;
__host__ __device__ constexpr int pf_ta_stages(int n_tile) { return (512 - (n_tile + 31) / 32 * 32) / PF_TA_STAGE_COLS < PF_TA_MAX_STAGES ? (512 - (n_tile + 31) / 32 * 32) / PF_TA_STAGE_COLS : PF_TA_MAX_STAGES; }

enum : int { PF_SMEM = 0, PF_TMEM = 1, PF_PAIR = 2 };   // where operand A goes; PF_PAIR: shared memory of two CTAs

struct PrefillArgs {
    const uint8_t* W;
    long long row_bytes;
    float* Y;
    long long ldy;
    int* status;
    int K, M, B, accumulate;
    int n_acc;             // accumulators in use per CTA: 1 or 2
    int n_tile;            // tokens per accumulator: a multiple of 16, at most 256
    int b_stages;
    int splits;            // CTAs of a cluster that share a tile's K
    int exact;             // Q4_K, Q5_K whose rows are only 2-byte aligned: no packed conversion
    const uint32_t* grid_src;
};

__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    // K-major, 128-byte swizzle: 8-row groups 1024 bytes apart (SBO), LBO unused (1), descriptor version 1
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// D format f32, A and B both bf16 (format code 1) or both fp16 (code 0), K-major, N = n_tile, M = 128
__device__ __forceinline__ uint32_t pf_idesc(bool f16, int n_tile) {
    return (1u << 4) | ((f16 ? 0u : 1u) << 7) | ((f16 ? 0u : 1u) << 10) | ((uint32_t)(n_tile >> 3) << 17) | ((uint32_t)(PF_ROWS >> 4) << 24);
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}

// the same, counted on a barrier of either CTA of a pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}

// ---------------------------------------------------------------------------------------------------------------
// Packed dequantization of the K-quants Q4_K, Q5_K, Q6_K to operand pairs.  An integer n < 128 becomes the bf16 number 128 + n by
// OR-ing it under the bit pattern 0x4300, the bias is subtracted exactly (bf16 holds every integer below 256), and one
// packed bf16 fused multiply-add applies scale and minimum to two weights.  Against the exact dequantizer the scale and
// the minimum are rounded to bf16 before instead of after the multiplication: a relative error of 2^-9 per weight, the
// same size as the rounding of the product to bf16 that the tensor core's operand format imposes anyway.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ __nv_bfloat162 u32_bf2(uint32_t v) { return *(const __nv_bfloat162*)&v; }
// The same for fp16 operands (the reference's prefill path multiplies fp16 weights, src/cuda/prefill.cu:30-85): an integer
// n < 1024 becomes the half 1024 + n under the bit pattern 0x6400.
struct OpBf16 {
    using V2 = __nv_bfloat162;
    static __device__ __forceinline__ V2 splat(float x) { return __float2bfloat162_rn(x); }
    static __device__ __forceinline__ V2 bias(int extra) { const uint32_t h = 0x4300u + (uint32_t)extra; const uint32_t v = h | (h << 16); return *(const V2*)&v; }
    static __device__ __forceinline__ void bytes(uint32_t t, V2 bs, V2& lo, V2& hi) {
        lo = __hsub2(u32_bf2(__byte_perm(t, 0x43434343u, 0x5140)), bs);
        hi = __hsub2(u32_bf2(__byte_perm(t, 0x43434343u, 0x5342)), bs);
    }
    static __device__ __forceinline__ uint32_t bits(V2 v) { return *(const uint32_t*)&v; }
};
struct OpF16 {
    using V2 = __half2;
    static __device__ __forceinline__ V2 splat(float x) { return __float2half2_rn(x); }
    static __device__ __forceinline__ V2 bias(int extra) { const uint32_t h = 0x6400u + (uint32_t)extra; const uint32_t v = h | (h << 16); return *(const V2*)&v; }   // 1024 + extra: one ulp = 1 up to 2047
    static __device__ __forceinline__ void bytes(uint32_t t, V2 bs, V2& lo, V2& hi) {
        const uint32_t l = __byte_perm(t, 0x64646464u, 0x5140), h = __byte_perm(t, 0x64646464u, 0x5342);
        lo = __hsub2(*(const V2*)&l, bs);
        hi = __hsub2(*(const V2*)&h, bs);
    }
    static __device__ __forceinline__ uint32_t bits(V2 v) { return *(const uint32_t*)&v; }
};

// p[j] = weights 2j, 2j + 1 of the sub-block; exact: multiplied in fp32 and rounded once whatever the format
template <int FMT, bool F16>
__device__ __forceinline__ void operand_pairs(const Sub32& o, bool exact, uint32_t (&p)[16]) {
    using OP = typename std::conditional<F16, OpF16, OpBf16>::type;
    using V2 = typename OP::V2;
    constexpr bool PACKED = FMT == T_Q4_K || FMT == T_Q5_K || FMT == T_Q6_K;
    if (PACKED && !exact) {
        const V2 bias = OP::bias(FMT == T_Q6_K ? 32 : 0);
        const V2 a0 = OP::splat(o.a[0]), a1 = FMT == T_Q6_K ? OP::splat(o.a[1]) : a0;
        const V2 c = OP::splat(FMT == T_Q6_K ? 0.0f : -o.c[0]);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            V2 lo, hi;
            OP::bytes(o.u[i], bias, lo, hi);
            const V2 a = i < 4 ? a0 : a1;
            p[2 * i] = FMT == T_Q6_K ? OP::bits(__hmul2(lo, a)) : OP::bits(__hfma2(lo, a, c));
            p[2 * i + 1] = FMT == T_Q6_K ? OP::bits(__hmul2(hi, a)) : OP::bits(__hfma2(hi, a, c));
        }
    } else {
#pragma unroll
        for (int j = 0; j < 16; j++) p[j] = sub32_pair<FMT, F16>(o, j);
    }
}

// true in one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_peer_f32(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// Arrives on a barrier of another CTA of the cluster.  (The weights it announces were made visible to the asynchronous proxy
// before, in the shared memory of the SM that holds them, where the tensor core reads them; release and acquire at cluster scope
// would add a memory fence of some 1800 clocks: 16384 x 5120 Q4_K, 1024 tokens 322 us against 138.)
__device__ __forceinline__ void mbar_arrive_peer(uint32_t addr) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory"); }
// the barrier is arrived on when the tensor core has done all that was issued before (both CTAs of a pair: in each of them)
template <bool PAIR>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    if constexpr (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 16 columns of this warp's 32 rows: 32 16-bit weights of a row
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 16 accumulator columns of this warp's 32 rows
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// F16: operands are fp16 (weights dequantized to fp16, activations fp16) instead of bf16.
// ALIGNED: every row starts at a multiple of expand_alignment(FMT).
// TA: operand A goes to tensor memory instead of shared memory (one accumulator: tiles of up to 256 tokens, also of longer
// calls that are cut so).  Up to there the kernel is
// bound by shared-memory bandwidth: per 128 K the tensor core reads 32 KB of weights and 20 KB of activations (80 tokens), the
// decode warps write the weights and move the raw blocks twice, 140 KB of traffic or 1100 clocks of some 1700 measured; from
// tensor memory the weights cost none of it.  With one wait and one commit per 128 K and the unchecked fetch, 16384 x 5120 Q4_K,
// 77 tokens 39.6 -> 27.9 us, 17408 x 5120 IQ3_XXS 51.4 -> 42.0, 5120 x 17408 Q6_K 55.1 -> 45.4, a Q4_K / Q6_K layer 199 -> 154 us.
// PAIR: two CTAs (a cluster of two, row tiles 2i and 2i + 1) multiply as one, M = 256 (cta_group::2): each expands its 128 rows and
// loads half of every activation tile, CTA 0 issues, each CTA's tensor memory holds its own rows.  For tiles over 256 tokens whose K is not
// shared, where there are two row tiles; alone a slab of 64 K moves 176 KB through an SM's shared memory (32 KB tiles written and read for each accumulator), 1375 clocks of
// which the tensor core needs 1024; in pairs 112 KB, and half the activation bytes from L2 (16384 x 5120 Q4_K,
// 1024 tokens 146 -> 132 us, 17408 x 5120 IQ3_XXS 161 -> 143; 512 tokens of the former 72 -> 66).
template <int FMT, bool F16, bool ALIGNED, int MODE>
__global__ void __launch_bounds__(PF_THREADS, 1) prefill_kernel(const PrefillArgs a, const __grid_constant__ CUtensorMap xmap) {
    constexpr bool TA = MODE == PF_TMEM, PAIR = MODE == PF_PAIR;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full_a = (uint64_t*)smem;              // [A stages] the 16 decode warps arrive
    constexpr int MAX_A = TA ? PF_TA_MAX_STAGES : PF_A_STAGES;
    const int a_stages = TA ? a.b_stages : PF_A_STAGES;
    uint64_t* empty_a = full_a + MAX_A;              // [A stages] tcgen05.commit
    uint64_t* full_b = empty_a + MAX_A;              // [B stages] TMA bytes
    uint64_t* empty_b = full_b + PF_B_MAX_STAGES;    // [B stages] tcgen05.commit
    uint64_t* acc_done = empty_b + PF_B_MAX_STAGES;  // [1]
    uint32_t* tmem_slot = (uint32_t*)(acc_done + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int b_stage_bytes = a.n_tile * (PF_KSLAB * 2) * (TA ? 2 : 1) / (PAIR ? 2 : 1);   // TA: a stage is 128 K of both operands, one barrier each way
    uint8_t* stages = smem + 1024;                                   // ring of weight tiles (TA: none)
    uint8_t* stages_b = stages + (TA ? 0 : PF_A_STAGES * PF_A_BYTES); // ring of activation tiles
    uint8_t* raw_all = stages_b + a.b_stages * b_stage_bytes;         // the decode warps' raw blocks
    uint32_t* tab_smem = (uint32_t*)(raw_all + (TA ? 2 * pf_raw_ta(FMT) : pf_raw_smem(FMT)));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = a.splits > 1 ? (int)cluster_rank() : 0;
    const int half_id = PAIR ? (int)cluster_rank() : 0;   // which CTA of the pair this is
    const int row0 = (int)(blockIdx.x / (unsigned)a.splits) * PF_ROWS;
    const int tile_tok = a.n_acc * a.n_tile;
    const int tok0 = blockIdx.y * tile_tok;
    const int nsb = a.K >> 8;
    const int sb_begin = nsb * rank / a.splits, sb_end = nsb * (rank + 1) / a.splits;   // this CTA's super-blocks (splits <= nsb: never none)
    const uint32_t tmem_cols = TA || a.n_acc == 2 ? 512u : a.n_tile > 128 ? 256u : a.n_tile > 64 ? 128u : a.n_tile > 32 ? 64u : 32u;

    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < a_stages; s++) {
            mbar_init(smem_u32(&full_a[s]), PF_DECODE_WARPS * (PAIR ? 2 : 1) + (TA ? 1 : 0));   // one arrival per warp (PAIR: of both CTAs, in CTA 0; TA: and the activations')
            mbar_init(smem_u32(&empty_a[s]), 1);
        }
        for (int s = 0; s < a.b_stages; s++) {
            mbar_init(smem_u32(&full_b[s]), 1);
            mbar_init(smem_u32(&empty_b[s]), 1);
        }
        mbar_init(smem_u32(acc_done), 1);
        mbar_fence_init();
    }
    if (warp == PF_DECODE_WARPS + 1) {   // this warp owns the tensor memory allocation
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    fill_grid_table<FMT>(tab_smem, a.grid_src, tid, PF_THREADS);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync_all();   // the other CTA's barriers are initialised
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    if (tid == 0 && (smem_u32(stages) & 1023u)) atomicOr(a.status, ST_TMEM_TIMEOUT);   // swizzled tiles need 1024-byte alignment

    if (warp < PF_DECODE_WARPS) {
        // ---------------- operand A: decode 128 rows x 128 weights per stage ----------------
        constexpr int RAW = pf_raw_bytes(FMT), PITCH = TA ? pf_pitch_ta(FMT, ALIGNED) : pf_pitch(FMT), ROUNDS = (pf_pieces(FMT) + 3) / 4;
        constexpr int UNIT_HALVES = FMT == T_Q8_0 ? 1 : 2;
        const uintptr_t w_begin = (uintptr_t)a.W, w_end = w_begin + (uintptr_t)(a.M - 1) * a.row_bytes + (uintptr_t)nsb * (RAW * 2 / UNIT_HALVES);
        // fetching: lane / 4 is the row, lane % 4 the first of its pieces; rows past the end repeat the last row (never stored)
        // (TA: the four warps of a quarter of the rows, warp % 4, fetch eight of its 32 rows each)
        const int first_row = TA ? 32 * (warp & 3) + PF_WARP_ROWS * (warp >> 2) : PF_WARP_ROWS * warp;
        const uintptr_t fetch_row = w_begin + (uintptr_t)min(row0 + first_row + (lane >> 2), a.M - 1) * a.row_bytes;
        uint8_t* raw = raw_all + first_row * PITCH;
        uint8_t* raw_put = raw + (lane >> 2) * PITCH + 16 * (lane & 3);
        // A piece that reaches past the matrix's first or last byte is not loaded ahead but copied by halfwords when it is due:
        // without that branch the loads stay in flight behind the work on the unit before (with it the compiler waited for
        // them on the spot).
        uint4 ahead[ROUNDS] = {};
        auto piece_at = [&](int unit, int r) { return ((fetch_row + (uintptr_t)unit * RAW) & ~(uintptr_t)15) + 16 * (uintptr_t)((lane & 3) + 4 * r); };
        auto inside = [&](uintptr_t at, int unit) { return at >= w_begin && at + 16 <= w_end && at < fetch_row + (uintptr_t)(unit + 1) * RAW; };
        // Every unit but the matrix's first and last: a piece is loaded where the unit can reach it at all, unchecked (it ends at
        // most 29 bytes past the unit, where the next one lies).  The checks alone were a third of a unit's instructions.
        const int row_first = min(row0 + first_row, a.M - 1), row_last = min(row0 + first_row + PF_WARP_ROWS - 1, a.M - 1), n_units = nsb * 2 / UNIT_HALVES;
        auto interior = [&](int unit) { return (row_first > 0 || unit > 0) && (row_last < a.M - 1 || unit + 1 < n_units); };
        auto reached = [&](int r) { return 4 * r + 3 < pf_pieces(FMT) || (lane & 3) + 4 * r < pf_pieces(FMT); };
        auto put_piece = [&](int r) {
            if constexpr (PITCH % 16 == 0) {
                *(uint4*)(raw_put + 64 * r) = ahead[r];
            } else {
                uint32_t* to = (uint32_t*)(raw_put + 64 * r);
                to[0] = ahead[r].x; to[1] = ahead[r].y; to[2] = ahead[r].z; to[3] = ahead[r].w;
            }
        };
        auto fetch = [&](int unit) {
            if (interior(unit)) {
                const uint8_t* at = (const uint8_t*)piece_at(unit, 0);
#pragma unroll
                for (int r = 0; r < ROUNDS; r++)
                    if (reached(r)) ahead[r] = __ldg((const uint4*)(at + 64 * r));
                return;
            }
#pragma unroll
            for (int r = 0; r < ROUNDS; r++) {
                const uintptr_t at = piece_at(unit, r);
                if (inside(at, unit)) ahead[r] = __ldg((const uint4*)at);
            }
        };
        auto put_raw = [&](int unit) {
            if (interior(unit)) {
#pragma unroll
                for (int r = 0; r < ROUNDS; r++)
                    if (reached(r)) put_piece(r);
                return;
            }
#pragma unroll
            for (int r = 0; r < ROUNDS; r++) {
                const uintptr_t at = piece_at(unit, r);
                if (inside(at, unit)) {
                    put_piece(r);
                } else if (at < fetch_row + (uintptr_t)(unit + 1) * RAW) {
                    for (int h = 0; h < 16; h += 2)
                        if (at + h >= w_begin && at + h < w_end) *(uint16_t*)(raw_put + 64 * r + h) = *(const uint16_t*)(at + h);
                }
            }
        };
        // expanding: lane % 8 is the row, lane / 8 the sub-block of the half super-block.  The eight rows of a quarter warp
        // store the same piece of their swizzled rows, which is eight different bank groups.
        // TA: a lane is a row of the warp's quarter, the warp's sub-block of the half is warp / 4.
        const int r7 = TA ? lane : lane & 7, q = TA ? warp >> 2 : lane >> 3;
        const uint32_t dec_lo = (uint32_t)w_begin + (uint32_t)min(row0 + (TA ? 32 * (warp & 3) : first_row) + r7, a.M - 1) * (uint32_t)a.row_bytes;
        const uint8_t* raw_get = raw_all + ((TA ? 32 * (warp & 3) : first_row) + r7) * PITCH;
        const uint32_t* tab = grid_copy<FMT>(tab_smem, lane);
        uint8_t* put = stages + (q >> 1) * PF_A_SLAB_BYTES + (PF_WARP_ROWS * warp + r7) * 128;
        const int unit_end = sb_end * 2 / UNIT_HALVES;
        const uint32_t a_tmem = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((a.n_tile + 31) / 32 * 32 + 16 * q);   // TA: this warp's columns of stage 0
        int st = 0, buf = 0;
        uint32_t use = 0;
        fetch(sb_begin * 2 / UNIT_HALVES);
        for (int unit = sb_begin * 2 / UNIT_HALVES; unit < unit_end; unit++) {
            put_raw(unit);
            if (TA) named_bar_sync(1 + (warp & 3), 128);   // (the buffer of two units before is free: its readers have come here since)
            else __syncwarp();
            if (unit + 1 < unit_end) fetch(unit + 1);
            const uint8_t* blk = raw_get + ((dec_lo + (uint32_t)unit * RAW) & 15u);
#pragma unroll
            for (int half = 0; half < UNIT_HALVES; half++) {
                Sub32 o;
                load_sub32<FMT, ALIGNED>(blk, 4 * half + q, tab, o);
                uint32_t p[16];
                operand_pairs<FMT, F16>(o, !ALIGNED && (FMT == T_Q4_K || FMT == T_Q5_K) && a.exact, p);
                mbar_wait_bounded(smem_u32(&empty_a[st]), use ^ 1u, abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT);
                if constexpr (TA) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    tmem_st16(a_tmem + (uint32_t)(st * PF_TA_STAGE_COLS), p);
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&full_a[st]));
                    if (++st == a_stages) { st = 0; use ^= 1u; }
                    continue;
                }
                // row of the tile: 128 bytes; 16-byte chunk c goes to chunk c ^ (row & 7) (128-byte swizzle)
                uint8_t* arow = put + st * PF_A_BYTES;
#pragma unroll
                for (int c = 0; c < 4; c++) *(uint4*)(arow + 16 * ((4 * (q & 1) + c) ^ r7)) = make_uint4(p[4 * c], p[4 * c + 1], p[4 * c + 2], p[4 * c + 3]);
                fence_proxy_async();                                 // generic-proxy stores -> visible to the tensor core
                __syncwarp();
                if (lane == 0) {
                    if (PAIR && half_id == 1) mbar_arrive_peer(peer_smem(smem_u32(&full_a[st]), 0u));
                    else mbar_arrive(smem_u32(&full_a[st]));
                }
                if (++st == PF_A_STAGES) { st = 0; use ^= 1u; }
            }
            if (TA) {   // the other buffer
                buf ^= 1;
                raw_put += buf ? pf_raw_ta(FMT) : -pf_raw_ta(FMT);
                raw_get += buf ? pf_raw_ta(FMT) : -pf_raw_ta(FMT);
            }
        }
    } else if (warp == PF_DECODE_WARPS) {
        // ---------------- operand B: activation tiles by TMA ----------------
        if (TA) {
            if (lane == 0) {
                int st = 0;
                uint32_t use = 0;
                for (int pair = 2 * sb_begin; pair < 2 * sb_end; pair++) {
                    mbar_wait_bounded(smem_u32(&empty_a[st]), use ^ 1u, abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT);
                    const uint32_t fb = smem_u32(&full_a[st]), to = smem_u32(stages_b + st * b_stage_bytes);
                    mbar_arrive_expect_tx(fb, (uint32_t)b_stage_bytes);
                    tma_load_2d(to, &xmap, 2 * pair * PF_KSLAB, tok0, fb);
                    tma_load_2d(to + (uint32_t)(b_stage_bytes / 2), &xmap, (2 * pair + 1) * PF_KSLAB, tok0, fb);
                    if (++st == a_stages) { st = 0; use ^= 1u; }
                }
            }
        } else if (lane == 0) {
            int st = 0;
            uint32_t use = 0;
            for (int slab = 4 * sb_begin; slab < 4 * sb_end; slab++)
                for (int n = 0; n < a.n_acc; n++) {
                    mbar_wait_bounded(smem_u32(&empty_b[st]), use ^ 1u, abort_flag, a.status, ST_WAIT_EMPTY_TIMEOUT);
                    const uint32_t fb = smem_u32(&full_b[st]), to = smem_u32(stages_b + st * b_stage_bytes);
                    if constexpr (PAIR) {   // both halves count on CTA 0's barrier
                        if (half_id == 0) mbar_arrive_expect_tx(fb, 2u * (uint32_t)b_stage_bytes);
                        tma_load_2d_pair(to, &xmap, slab * PF_KSLAB, tok0 + n * a.n_tile + half_id * (a.n_tile / 2), peer_smem(fb, 0u));
                    } else {
                        mbar_arrive_expect_tx(fb, (uint32_t)b_stage_bytes);
                        tma_load_2d(to, &xmap, slab * PF_KSLAB, tok0 + n * a.n_tile, fb);
                    }
                    if (++st == a.b_stages) { st = 0; use ^= 1u; }
                }
        }
    } else {
        // ---------------- MMA issue ----------------
        // The whole warp walks the rings and one elected lane issues: descriptors, addresses and counts are then the same in
        // every lane and stay in uniform registers.  (Under `if (lane == 0)` an MMA took about 250 clocks to issue, four
        // times what the tensor core needs for 16 tokens: 16384 x 5120 Q4_K, 16 tokens 62 -> 40 us.)
        const uint32_t idesc = pf_idesc(F16, a.n_tile) + (PAIR ? (uint32_t)(PF_ROWS >> 4) << 24 : 0u);   // PAIR: M = 256
        const uint64_t desc0 = umma_desc_sw128(0);
        const uint32_t a_lo = (smem_u32(stages) & 0x3FFFFu) >> 4, b_lo = (smem_u32(stages_b) & 0x3FFFFu) >> 4;
        const uint32_t a_tmem = tmem_base + (uint32_t)((a.n_tile + 31) / 32 * 32);   // TA: A stages behind the accumulator
        int sa = 0, sb = 0;
        uint32_t use_a = 0, use_b = 0, accum = 0;
        if constexpr (TA) {
            // One wait, eight MMA and one commit per 128 K: with a wait and a commit per 64 K and operand this warp set the pace
            // (16384 x 5120 Q4_K, 16 or 77 tokens: 1300 clocks per 128 K, of which the tensor core needs 200 to 430).
            for (int pair = 2 * sb_begin; pair < 2 * sb_end; pair++) {
                mbar_wait_bounded(smem_u32(&full_a[sa]), use_a, abort_flag, a.status, ST_WAIT_FULL_TIMEOUT);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t bdesc = desc0 + (b_lo + (uint32_t)((sa * b_stage_bytes) >> 4));
                const uint32_t at = a_tmem + (uint32_t)(sa * PF_TA_STAGE_COLS), half_b = (uint32_t)(b_stage_bytes >> 5);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        asm volatile(
                            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                            ::"r"(tmem_base), "r"(at + (uint32_t)(8 * k)), "l"(bdesc + (uint64_t)((k >> 2) * half_b + 2 * (k & 3))), "r"(idesc),
                              "r"(k > 0 ? 1u : accum)
                            : "memory");
                    umma_commit<false>(smem_u32(&empty_a[sa]));
                }
                __syncwarp();
                accum = 1u;
                if (++sa == a_stages) { sa = 0; use_a ^= 1u; }
            }
        } else if (!(PAIR && half_id == 1))   // (CTA 0 of a pair issues for both)
        for (int pair = 2 * sb_begin; pair < 2 * sb_end; pair++) {
            mbar_wait_bounded(smem_u32(&full_a[sa]), use_a, abort_flag, a.status, ST_WAIT_FULL_TIMEOUT);
#pragma unroll
            for (int slab = 0; slab < 2; slab++) {
                const uint64_t adesc = desc0 + (a_lo + (uint32_t)((sa * PF_A_BYTES + slab * PF_A_SLAB_BYTES) >> 4));
                for (int n = 0; n < a.n_acc; n++) {
                    mbar_wait_bounded(smem_u32(&full_b[sb]), use_b, abort_flag, a.status, ST_WAIT_FULL_TIMEOUT);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bdesc = desc0 + (b_lo + (uint32_t)((sb * b_stage_bytes) >> 4));
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < PF_KSLAB / 16; k++) {
                            const uint32_t to = tmem_base + (uint32_t)(n * PF_MAX_N), add = k > 0 ? 1u : accum;
                            if constexpr (PAIR)
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(to), "l"(adesc + (uint64_t)(2 * k)),
                                    "l"(bdesc + (uint64_t)(2 * k)), "r"(idesc), "r"(add)
                                    : "memory");
                            else
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(to), "l"(adesc + (uint64_t)(2 * k)),
                                    "l"(bdesc + (uint64_t)(2 * k)), "r"(idesc), "r"(add)
                                    : "memory");
                        }
                        // frees the stages once the tensor core has read them (PAIR: in both CTAs)
                        umma_commit<PAIR>(smem_u32(&empty_b[sb]));
                        if (slab == 1 && n == a.n_acc - 1) umma_commit<PAIR>(smem_u32(&empty_a[sa]));
                    }
                    __syncwarp();
                    if (++sb == a.b_stages) { sb = 0; use_b ^= 1u; }
                }
                accum = 1u;
            }
            if (++sa == a_stages) { sa = 0; use_a ^= 1u; }
        }
        if (!(PAIR && half_id == 1) && elect_one()) umma_commit<PAIR>(smem_u32(acc_done));
        __syncwarp();
    }

    // ---------------- epilogue: warp w reads the accumulators' lanes 32 (w % 4) .. + 31, 16 tokens at a time ----------------
    const int n_tok = min(tile_tok, a.B - tok0), n_chunks = (n_tok + 15) >> 4;
    const int quad = warp & 3, row = row0 + 32 * quad + lane;
    auto acc_addr = [&](int chunk) {   // chunk of 16 tokens of the tile; an accumulator holds n_tile of them
        const int t = 16 * chunk, acc = t >= a.n_tile ? 1 : 0;
        return tmem_base + ((uint32_t)(32 * quad) << 16) + (uint32_t)(acc * PF_MAX_N + t - acc * a.n_tile);
    };
    auto store = [&](int chunk, const float (&v)[16]) {
        if (row >= a.M) return;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int t = 16 * chunk + j;
            if (t < n_tok) {
                float* yo = a.Y + (size_t)(tok0 + t) * a.ldy + row;
                *yo = a.accumulate ? *yo + v[j] : v[j];
            }
        }
    };
    if (warp < PF_DECODE_WARPS) {
        mbar_wait_bounded(smem_u32(acc_done), 0u, abort_flag, a.status, ST_TMEM_TIMEOUT);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (a.splits == 1) {
        if (warp < PF_DECODE_WARPS)
            for (int chunk = warp >> 2; chunk < n_chunks; chunk += PF_DECODE_WARPS / 4) {
                uint32_t v[16];
                float f[16];
                tmem_ld16(acc_addr(chunk), v);
#pragma unroll
                for (int j = 0; j < 16; j++) f[j] = __uint_as_float(v[j]);
                store(chunk, f);
            }
    } else {
        // Chunk c of the tile is finished by rank c % splits: the others put their sums of it into that CTA's (now idle)
        // rings, [source][c / splits][16 tokens][128 rows], sources in rank order without the owner.
        const int own_chunks = (n_chunks + a.splits - 1) / a.splits;
        const uint32_t ring = smem_u32(stages);
        cluster_sync_all();                                  // every CTA's tensor core has read its rings
        if (warp < PF_DECODE_WARPS)
            for (int chunk = warp >> 2; chunk < n_chunks; chunk += PF_DECODE_WARPS / 4) {
                const int owner = chunk % a.splits;
                if (owner == rank) continue;
                uint32_t v[16];
                tmem_ld16(acc_addr(chunk), v);
                const int src = rank - (rank > owner ? 1 : 0);
                const uint32_t dst = peer_smem(ring + (uint32_t)((src * own_chunks + chunk / a.splits) * (16 * PF_ROWS) + 32 * quad + lane) * 4u, (uint32_t)owner);
#pragma unroll
                for (int j = 0; j < 16; j++) st_peer_f32(dst + (uint32_t)(j * PF_ROWS * 4), v[j]);
            }
        cluster_sync_all();                                  // all sums have arrived; nobody touches another CTA's memory after this
        if (warp < PF_DECODE_WARPS)
            for (int own = warp >> 2; own * a.splits + rank < n_chunks; own += PF_DECODE_WARPS / 4) {
                uint32_t v[16];
                float f[16];
                tmem_ld16(acc_addr(own * a.splits + rank), v);
#pragma unroll
                for (int j = 0; j < 16; j++) f[j] = 0.0f;
                for (int r = 0; r < a.splits; r++) {
                    if (r == rank) {
#pragma unroll
                        for (int j = 0; j < 16; j++) f[j] += __uint_as_float(v[j]);
                        continue;
                    }
                    const float* in = (const float*)stages + (size_t)((r - (r > rank ? 1 : 0)) * own_chunks + own) * (16 * PF_ROWS) + 32 * quad + lane;
#pragma unroll
                    for (int j = 0; j < 16; j++) f[j] += in[j * PF_ROWS];
                }
                store(own * a.splits + rank, f);
            }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (PAIR) cluster_sync_all();   // the allocation is both CTAs': neither gives it back before the other's last read
    else __syncthreads();
    if (warp == PF_DECODE_WARPS + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
    if (PAIR) cluster_sync_all();   // neither CTA leaves before both have given it back
}


typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// How a GEMM is cut: token tiles of n_acc x n_tile tokens and K shared by `splits` CTAs.
struct PrefillCut { int n_acc, n_tile, tok_tiles, splits, b_stages, mode; };

// what a CTA receives from the others of its cluster (over the rings, idle by then; operand A in tensor memory: and what follows)
int exchange_bytes(const PrefillCut& c) { return (c.splits - 1) * ((c.n_acc * c.n_tile / 16 + c.splits - 1) / c.splits) * (16 * PF_ROWS * 4); }

// Clocks in which the expanders of a format bring 128 rows x 64 K into tensor memory
double expand_clocks(int fmt) {
    switch (fmt) {
        case T_Q4_K: return 460.0;
        case T_Q5_K: return 570.0;
        case T_Q2_K: return 615.0;
        case T_IQ1_S: return 645.0;
        case T_IQ2_XXS: return 705.0;
        case T_IQ2_XS: case T_IQ1_M: return 725.0;
        case T_IQ2_S: return 745.0;
        case T_IQ3_S: case T_IQ3_XXS: return 790.0;
        case T_Q6_K: return 820.0;
        case T_Q8_0: return 875.0;
        default: return 940.0;   // IQ4_XS
    }
}
// Picks the cut by its time in SM clocks: rounds of CTAs over the SMs, a K-slab at a time.  A slab takes the longer of what its
// expanders and what its tokens take, added as fourth powers: the format's clocks against 2.5 a token with operand A in tensor memory,
// 0.6 of them and 710 against 1.65 a token in pairs, 0.47 of them and 1000 against 2.3 with operand A in shared memory (their swizzled
// stores and barriers are the same for every format).  10400 clocks start a CTA and drain it, 30 per token store the tile; a cluster's
// exchange costs 500 and another 1.4 per token.  Clusters of three and more leave some SMs of a GPC unused (at M = 5120, 120 CTAs in threes
// take 60 us where 160 in fours, 132 of which fit at once, take 88), those of seven and eight more of them (2048 x 4096 IQ2_XS, 77
// tokens: 128 CTAs in eights 21.8 us, 96 in sixes 14.4).  The constants are fitted to every cut of as many to twice as many token tiles
// and up to eight CTAs over 1547 calls (thirteen formats, twelve shapes, 16 to 2500 tokens): the cut picked takes 0.3 % more than the
// fastest on average and over 5 % more in 42 of them; with one set of constants for all formats, measured on Q4_K, it was 3.7 % and 324
// (5120 x 17408 on 1024 tokens, IQ4_XS 195 us in pairs, 184 in threes).  M = 5120, K = 17408, IQ4_XS, 512 tokens: 277 us unsplit, 101 us in threes.
bool prefill_cut(const q38b_ctx* ctx, int fmt, int K, int M, int B, PrefillCut* best) {
    const long long row_tiles = (M + PF_ROWS - 1) / PF_ROWS;
    const int nsb = K / 256;
    double best_cost = 0.0;
    bool found = false;
    const int min_tiles = (B + 2 * PF_MAX_N - 1) / (2 * PF_MAX_N);
    for (int want = min_tiles; want <= 2 * min_tiles + 1; want++) {
        const int per = (B + want - 1) / want;
        PrefillCut c;
        c.n_acc = per > PF_MAX_N ? 2 : 1;
        const int step = c.n_acc == 2 ? 32 : 16;   // (in pairs each CTA loads half of a tile)
        c.n_tile = ((per + c.n_acc - 1) / c.n_acc + step - 1) / step * step;
        const int tile = c.n_acc * c.n_tile;
        c.tok_tiles = (B + tile - 1) / tile;
        if (ctx->prefill_tiles && want != ctx->prefill_tiles) continue;
        const bool ta = c.n_acc == 1;
        const int room = ctx->smem_optin - pf_fixed_smem(fmt, ta);
        const int stage = c.n_tile * PF_KSLAB * 2 * (ta ? 2 : 1);
        if (room / stage < 2) continue;
        for (c.splits = 1; c.splits <= std::min(PF_MAX_SPLITS, nsb); c.splits++) {
            if (ctx->prefill_splits && c.splits != ctx->prefill_splits) continue;
            c.mode = ta ? PF_TMEM : c.splits == 1 && row_tiles > 1 ? PF_PAIR : PF_SMEM;
            c.b_stages = std::min(ta ? pf_ta_stages(c.n_tile) : PF_B_MAX_STAGES, room / (c.mode == PF_PAIR ? stage / 2 : stage));
            if (ta ? 1024 + exchange_bytes(c) > ctx->smem_optin : exchange_bytes(c) > PF_A_STAGES * PF_A_BYTES + c.b_stages * stage) continue;
            const long long ctas = (c.mode == PF_PAIR ? (row_tiles + 1) / 2 * 2 : row_tiles) * c.tok_tiles * c.splits;
            const int slots = c.splits <= 2 ? ctx->sm_count : (c.splits <= 6 ? ctx->sm_count * 9 / 10 : ctx->sm_count * 3 / 4) / c.splits * c.splits;
            const double rounds = (double)((ctas + slots - 1) / slots);
            const double expand = c.mode == PF_TMEM ? expand_clocks(fmt) : c.mode == PF_PAIR ? 710.0 + 0.6 * expand_clocks(fmt) : 1000.0 + 0.47 * expand_clocks(fmt);
            const double multiply = (c.mode == PF_PAIR ? 1.65 : ta ? 2.5 : 2.3) * tile, e2 = expand * expand, m2 = multiply * multiply;
            const double slab = std::sqrt(std::sqrt(e2 * e2 + m2 * m2));
            const double cost = rounds * (4.0 * ((nsb + c.splits - 1) / c.splits) * slab + 10400.0 + 30.0 * tile + (c.splits > 1 ? 500.0 + 1.4 * tile : 0.0));
            if (!found || cost < best_cost) { found = true; best_cost = cost; *best = c; }
        }
    }
    return found;
}

template <int FMT, bool F16, bool ALIGNED, int MODE>
int launch_prefill_as(q38b_ctx* ctx, const PrefillArgs& a, const CUtensorMap& map, const PrefillCut& cut, cudaStream_t st) {
    constexpr bool TA = MODE == PF_TMEM, PAIR = MODE == PF_PAIR;
    auto kern = prefill_kernel<FMT, F16, ALIGNED, MODE>;
    bool known = false;   // opt-in shared-memory size: once per context (= device) and kernel
    for (int i = 0; i < ctx->n_configured; i++) known |= ctx->configured[i] == (const void*)kern;
    if (!known) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin);
        if (e != cudaSuccess) { ctx->last_cuda = (int)e; return Q38B_ERR_CUDA; }
        if (ctx->n_configured < (int)(sizeof(ctx->configured) / sizeof(ctx->configured[0]))) ctx->configured[ctx->n_configured++] = (const void*)kern;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    const int row_tiles = (a.M + PF_ROWS - 1) / PF_ROWS;
    cfg.gridDim = dim3((unsigned)(PAIR ? (row_tiles + 1) / 2 * 2 : row_tiles * cut.splits), (unsigned)cut.tok_tiles);
    cfg.blockDim = dim3(PF_THREADS);
    cfg.dynamicSmemBytes = (size_t)std::max(pf_fixed_smem(FMT, TA) + cut.b_stages * (cut.n_tile * PF_KSLAB * 2 * (TA ? 2 : 1) / (PAIR ? 2 : 1)), TA ? 1024 + exchange_bytes(cut) : 0);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = PAIR ? 2u : (unsigned)cut.splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = PAIR || cut.splits > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a, map);
    if (e != cudaSuccess) { (void)cudaGetLastError(); ctx->last_cuda = (int)e; return Q38B_ERR_CUDA; }
    return Q38B_OK;
}

template <int FMT, bool F16, bool ALIGNED>
int launch_prefill_op(q38b_ctx* ctx, const PrefillArgs& a, const CUtensorMap& map, const PrefillCut& cut, cudaStream_t st) {
    switch (cut.mode) {
        case PF_TMEM: return launch_prefill_as<FMT, F16, ALIGNED, PF_TMEM>(ctx, a, map, cut, st);
        case PF_PAIR: return launch_prefill_as<FMT, F16, ALIGNED, PF_PAIR>(ctx, a, map, cut, st);
        default: return launch_prefill_as<FMT, F16, ALIGNED, PF_SMEM>(ctx, a, map, cut, st);
    }
}

template <int FMT>
int launch_prefill(q38b_ctx* ctx, PrefillArgs a, const CUtensorMap& map, const PrefillCut& cut, cudaStream_t st, bool f16) {
    if constexpr (expand_alignment(FMT) > 2) {
        constexpr int AL = expand_alignment(FMT) - 1;
        if ((((uintptr_t)a.W | (uintptr_t)a.row_bytes) & AL) == 0)
            return f16 ? launch_prefill_op<FMT, true, true>(ctx, a, map, cut, st) : launch_prefill_op<FMT, false, true>(ctx, a, map, cut, st);
    }
    return f16 ? launch_prefill_op<FMT, true, false>(ctx, a, map, cut, st) : launch_prefill_op<FMT, false, false>(ctx, a, map, cut, st);
}

int gemm_prefill_any(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int M, const void* X, long long ldx, int B,
                     float* Y, long long ldy, int accumulate, void* stream, bool f16) {
    if (!ctx || !W || !X || !Y || K <= 0 || K % 256 || M < 1 || B < 1 || ldx < K || ldy < M) return Q38B_ERR_ARG;
    if (!q38b_format_supported(type)) return Q38B_ERR_UNSUPPORTED;
    if (row_bytes < q38b_row_bytes(type, K)) return Q38B_ERR_ARG;
    if (((uintptr_t)W & 1) || (row_bytes & 1) || ((uintptr_t)X & 15) || ((ldx * 2) & 15) || ((uintptr_t)Y & 3)) return Q38B_ERR_ALIGN;
    EncodeTiledFn enc = encode_fn();
    if (!enc) return Q38B_ERR_UNSUPPORTED;
    PrefillCut cut;
    if (!prefill_cut(ctx, (int)type, K, M, B, &cut)) return Q38B_ERR_NOMEM;
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)B};
    const cuuint64_t strides[1] = {(cuuint64_t)ldx * 2};
    const cuuint32_t box[2] = {PF_KSLAB, (cuuint32_t)(cut.mode == PF_PAIR ? cut.n_tile / 2 : cut.n_tile)};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)X, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return Q38B_ERR_ARG;
    PrefillArgs a;
    a.W = (const uint8_t*)W;
    a.row_bytes = (long long)row_bytes;
    a.Y = Y;
    a.ldy = ldy;
    a.status = ctx->d_status;
    a.K = K;
    a.M = M;
    a.B = B;
    a.accumulate = accumulate ? 1 : 0;
    a.n_acc = cut.n_acc;
    a.n_tile = cut.n_tile;
    a.b_stages = cut.b_stages;
    a.splits = cut.splits;
    a.grid_src = q38b_grid_source(ctx, type);
    a.exact = (((uintptr_t)W | row_bytes) & 3) != 0;   // such rows have always been multiplied exactly
    cudaStream_t st = (cudaStream_t)stream;
    switch (type) {
#define Q38B_CASE(T) case T: return launch_prefill<T>(ctx, a, map, cut, st, f16)
        Q38B_CASE(T_Q8_0); Q38B_CASE(T_Q4_K); Q38B_CASE(T_Q5_K); Q38B_CASE(T_Q6_K); Q38B_CASE(T_IQ3_XXS); Q38B_CASE(T_IQ3_S); Q38B_CASE(T_IQ4_XS);
        Q38B_CASE(T_Q2_K); Q38B_CASE(T_IQ2_XXS); Q38B_CASE(T_IQ2_XS); Q38B_CASE(T_IQ2_S); Q38B_CASE(T_IQ1_S); Q38B_CASE(T_IQ1_M);
#undef Q38B_CASE
        default: return Q38B_ERR_UNSUPPORTED;
    }
}

}  // namespace

// Test hook (not in the public header): the cut of a GEMM on a 148-SM device with 227 KB of shared memory a CTA, no device needed: token
// tiles, tokens a tile, CTAs that share K, where operand A goes (0 shared memory, 1 tensor memory, 2 a pair's shared memory).
extern "C" int q38b_debug_prefill_plan(uint32_t type, int K, int M, int B, int* out) {
    q38b_ctx ctx;
    ctx.sm_count = 148;
    ctx.smem_optin = 232448;
    PrefillCut c;
    if (!prefill_cut(&ctx, (int)type, K, M, B, &c)) return Q38B_ERR_NOMEM;
    const int v[4] = {c.tok_tiles, c.n_acc * c.n_tile, c.splits, c.mode};
    memcpy(out, v, sizeof(v));
    return Q38B_OK;
}

// Test hook (not in the public header): the prefill GEMM cuts the tokens into `tiles` tiles and shares a tile's K among
// `splits` CTAs (0: its own rule), so that tests reach every cut with small matrices.
extern "C" int q38b_debug_set_prefill_cut(q38b_ctx* ctx, int tiles, int splits) {
    if (!ctx || tiles < 0 || splits < 0 || splits > PF_MAX_SPLITS) return Q38B_ERR_ARG;
    ctx->prefill_tiles = tiles;
    ctx->prefill_splits = splits;
    return Q38B_OK;
}

extern "C" int q38b_gemm_prefill(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int M, const void* X,
                                 long long ldx, int B, float* Y, long long ldy, int accumulate, void* stream) {
    return gemm_prefill_any(ctx, type, W, row_bytes, K, M, X, ldx, B, Y, ldy, accumulate, stream, false);
}

extern "C" int q38b_gemm_prefill_f16(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int M, const void* X,
                                     long long ldx, int B, float* Y, long long ldy, int accumulate, void* stream) {
    return gemm_prefill_any(ctx, type, W, row_bytes, K, M, X, ldx, B, Y, ldy, accumulate, stream, true);
}
