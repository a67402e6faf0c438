// q38b_dequant.cu -- rows of GGUF blocks written out as dense fp32 / fp16 / bf16 (q38b_dequant_rows).
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/q38b200.h"
#include "q38b_expand.cuh"
#include "q38b_internal.h"

using namespace q38b;

namespace {

// One warp per slice of 1024 weights, lane = sub-block of 32.  Bound by HBM: 0.4 bytes read and 2 (fp32: 4) written per
// weight.  The raw bytes come in as 16-byte pieces (one coalesced load instruction per 512 bytes, the next slice's in
// flight while this one is worked on), the results go through shared memory so that a warp stores 512 consecutive bytes.
// 17408 x 5120 IQ3_XXS to fp16 (212 MB): 43.6 us = 4.9 TB/s, against 558 us with one thread per sub-block reading single
// bytes and storing its own 64-byte run; the thirteen formats take 40-51 us to 16 bits (4.6-5.4 TB/s), 72-82 us to fp32.
// warps of a CTA and resident CTAs per SM: 64 registers a thread (fp32: 80), at most 42 KB of shared memory a CTA
__host__ __device__ constexpr int dq_warps(int kind) { return kind == Q38B_OUT_F32 ? 4 : 8; }
__host__ __device__ constexpr int dq_ctas(int kind) { return kind == Q38B_OUT_F32 ? 6 : 4; }
constexpr int DQ_RAW_BYTES = 4 * 272 + 16 + 16;  // the largest slice (Q8_0), its alignment, and what aligned word loads read past it

template <int FMT, int KIND>
__global__ void __launch_bounds__(dq_warps(KIND) * 32, dq_ctas(KIND)) dequant_rows_kernel(const uint8_t* __restrict__ W, long long row_bytes, int K, int rows,
                                                                              const uint32_t* __restrict__ grid_src, uint8_t* __restrict__ out) {
    constexpr int DQ_WARPS = dq_warps(KIND);
    constexpr int BB = Unit<FMT>::BLOCK_BYTES;
    constexpr int ESIZE = KIND == Q38B_OUT_F32 ? 4 : 2;
    constexpr int CHUNKS = 32 * ESIZE / 16;      // 16-byte pieces of a lane's 32 results
    constexpr int PIECES = (4 * BB + 15 + 15) / 16, ROUNDS = (PIECES + 31) / 32;
    __shared__ __align__(16) uint8_t raw_smem[DQ_WARPS][DQ_RAW_BYTES];
    __shared__ __align__(16) uint8_t out_smem[DQ_WARPS][1024 * ESIZE];
    __shared__ __align__(16) uint32_t tab_smem[grid_table_bytes(FMT) / 4 + 4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nsb = K >> 8, n_slices = (nsb + 3) >> 2;
    const uint32_t n_ctas = gridDim.x;
    const int step_row = (int)(n_ctas * DQ_WARPS / (uint32_t)n_slices), step_sl = (int)(n_ctas * DQ_WARPS % (uint32_t)n_slices);
    const uintptr_t w_begin = (uintptr_t)W, w_end = w_begin + (uintptr_t)(rows - 1) * row_bytes + (uintptr_t)nsb * BB;

    uint4 ahead[ROUNDS];
    auto fetch = [&](int row, int sl) {
        const uintptr_t src = w_begin + (uintptr_t)row * row_bytes + (uintptr_t)sl * (4 * BB);
        const uintptr_t end = src + (uintptr_t)min(4, nsb - 4 * sl) * BB, lo = src & ~(uintptr_t)15;
#pragma unroll
        for (int r = 0; r < ROUNDS; r++) {
            const uintptr_t at = lo + 16 * (uintptr_t)(lane + 32 * r);
            ahead[r] = make_uint4(0u, 0u, 0u, 0u);
            if (at >= end) continue;
            if (at >= w_begin && at + 16 <= w_end) {
                ahead[r] = __ldg((const uint4*)at);
            } else {                             // the matrix starts or ends inside this 16-byte unit
                uint32_t v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int h = 0; h < 8; h++)
                    if (at + 2 * h >= w_begin && at + 2 * h < w_end) v[h >> 1] |= (uint32_t)*(const uint16_t*)(at + 2 * h) << (16 * (h & 1));
                ahead[r] = make_uint4(v[0], v[1], v[2], v[3]);
            }
        }
    };
    // this warp's slices: every (CTAs x warps)-th one, stepped as (row, slice)
    const uint32_t first = blockIdx.x * DQ_WARPS + (uint32_t)warp;
    int row = (int)(first / (uint32_t)n_slices), sl = (int)(first % (uint32_t)n_slices);
    if (row < rows) fetch(row, sl);
    fill_grid_table<FMT>(tab_smem, grid_src, (int)threadIdx.x, DQ_WARPS * 32);
    __syncthreads();
    const uint32_t* tab = grid_copy<FMT>(tab_smem, lane);
    uint8_t* raw = raw_smem[warp];
    uint8_t* stage = out_smem[warp];
    const bool out_aligned = ((uintptr_t)out & 15) == 0;
    while (row < rows) {
        int next_row = row + step_row, next_sl = sl + step_sl;
        if (next_sl >= n_slices) { next_sl -= n_slices; next_row++; }
        const int mis = (int)((w_begin + (uintptr_t)row * row_bytes + (uintptr_t)sl * (4 * BB)) & 15);
        const int sb_here = min(4, nsb - 4 * sl);
#pragma unroll
        for (int r = 0; r < ROUNDS; r++)
            if (lane + 32 * r < PIECES) *(uint4*)(raw + 16 * (lane + 32 * r)) = ahead[r];
        __syncwarp();
        if (next_row < rows) fetch(next_row, next_sl);
        if ((lane >> 3) < sb_here) {
            Sub32 o;
            load_sub32<FMT, false>(raw + mis + BB * (lane >> 3), lane & 7, tab, o);
            // piece c of lane l is piece l * CHUNKS + c of the slice; it is kept at a place rotated within its group of eight (or
            // four), so that neither these stores nor the loads below meet on a bank
#pragma unroll
            for (int c = 0; c < CHUNKS; c++) {
                uint32_t v[4];
                if constexpr (KIND == Q38B_OUT_F32) {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int k = 4 * c + i;
                        v[i] = __float_as_uint(sub32_value<FMT>(o, k));
                        if (expand_form(FMT) == FORM_MAGNITUDE) v[i] ^= (o.sign << (31 - k)) & 0x80000000u;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++) v[i] = sub32_pair<FMT, KIND == Q38B_OUT_F16>(o, 4 * c + i);
                }
                const int piece = lane * CHUNKS + c;
                *(uint4*)(stage + 16 * (piece ^ ((piece >> 3) & (CHUNKS - 1)))) = make_uint4(v[0], v[1], v[2], v[3]);
            }
        }
        __syncwarp();
        uint8_t* dst = out + ((size_t)row * K + (size_t)sl * 1024) * ESIZE;
#pragma unroll
        for (int c = 0; c < CHUNKS; c++) {
            const int piece = lane + 32 * c;
            if (piece >= sb_here * 8 * CHUNKS) continue;
            const uint4 v = *(const uint4*)(stage + 16 * (piece ^ ((piece >> 3) & (CHUNKS - 1))));
            if (out_aligned) {
                __stcs((uint4*)(dst + 16 * piece), v);
            } else {
                uint32_t* d = (uint32_t*)(dst + 16 * piece);
                d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
            }
        }
        __syncwarp();
        row = next_row;
        sl = next_sl;
    }
}

template <int KIND>
int launch(q38b_ctx* ctx, uint32_t type, const uint8_t* W, long long rb, int K, int rows, uint8_t* out, cudaStream_t st) {
    const long long units = (long long)rows * ((K / 256 + 3) / 4);
    constexpr int warps = dq_warps(KIND);
    const unsigned blocks = (unsigned)std::min<long long>((units + warps - 1) / warps, (long long)ctx->sm_count * dq_ctas(KIND));
    const uint32_t* src = q38b_grid_source(ctx, type);
    switch (type) {
#define Q38B_CASE(T) case T: dequant_rows_kernel<T, KIND><<<blocks, warps * 32, 0, st>>>(W, rb, K, rows, src, out); break
        Q38B_CASE(T_Q8_0); Q38B_CASE(T_Q4_K); Q38B_CASE(T_Q5_K); Q38B_CASE(T_Q6_K); Q38B_CASE(T_IQ3_XXS); Q38B_CASE(T_IQ3_S); Q38B_CASE(T_IQ4_XS);
        Q38B_CASE(T_Q2_K); Q38B_CASE(T_IQ2_XXS); Q38B_CASE(T_IQ2_XS); Q38B_CASE(T_IQ2_S); Q38B_CASE(T_IQ1_S); Q38B_CASE(T_IQ1_M);
#undef Q38B_CASE
        default: return Q38B_ERR_UNSUPPORTED;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ctx->last_cuda = (int)e; return Q38B_ERR_CUDA; }
    return Q38B_OK;
}

}  // namespace

extern "C" int q38b_dequant_rows(q38b_ctx* ctx, uint32_t type, const void* W, size_t row_bytes, int K, int rows, void* out, int out_kind, void* stream) {
    if (!ctx || !W || !out || K <= 0 || K % 256 || rows < 1) return Q38B_ERR_ARG;
    if (!q38b_format_supported(type)) return Q38B_ERR_UNSUPPORTED;
    if (row_bytes < q38b_row_bytes(type, K)) return Q38B_ERR_ARG;
    if (((uintptr_t)W & 1) || (row_bytes & 1) || ((uintptr_t)out & 3)) return Q38B_ERR_ALIGN;
    cudaStream_t st = (cudaStream_t)stream;
    switch (out_kind) {
        case Q38B_OUT_F32: return launch<Q38B_OUT_F32>(ctx, type, (const uint8_t*)W, (long long)row_bytes, K, rows, (uint8_t*)out, st);
        case Q38B_OUT_F16: return launch<Q38B_OUT_F16>(ctx, type, (const uint8_t*)W, (long long)row_bytes, K, rows, (uint8_t*)out, st);
        case Q38B_OUT_BF16: return launch<Q38B_OUT_BF16>(ctx, type, (const uint8_t*)W, (long long)row_bytes, K, rows, (uint8_t*)out, st);
        default: return Q38B_ERR_ARG;
    }
}
