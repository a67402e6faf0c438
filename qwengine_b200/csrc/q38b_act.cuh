// q38b_act.cuh -- activation-side kernels: the quantizers, SwiGLU, residual add + RMSNorm, the bf16 matvec.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdint>

#include "q38b_decode.cuh"
#include "q38b_pipe.cuh"

namespace q38b {

#define Q38B_CODEBOOK_QUALIFIER __device__ const
#include "codebooks.inc"
#undef Q38B_CODEBOOK_QUALIFIER

// Two and four int32 values saturated to int8 and packed (cvt.pack: low byte = the last operand of each pair).
__device__ __forceinline__ uint32_t pack_s8x4(int q0, int q1, int q2, int q3) {
    uint32_t hi, w;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(q3), "r"(q2), "r"(0));
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q1), "r"(q0), "r"(hi));
    return w;
}

// One warp turns 256 floats, eight per lane (lane l: elements 8l .. 8l+7), into the values of a ggml Q8_K block.
// Arithmetic of quantize_row_q8_K_ref (src/quant/quant_ref.cpp:353-381): the FIRST element of largest magnitude, with
// its sign, maps to -127 (iscale = -127 / that element); q = min(127, round-half-even(iscale * x)); d = 1 / iscale; a
// block of zeros stays all zero.  Outputs: this lane's eight int8 values packed in w0 | w1, their sum s8, and d (the
// same in every lane).
__device__ __forceinline__ void q8k_block_core(const float (&v)[8], uint32_t& w0, uint32_t& w1, int& s8, float& d) {
    // Magnitudes compare like their bit patterns, so the block maximum is an integer maximum: one REDUX over the warp.
    uint32_t mag[8], lane_top = 0;
#pragma unroll
    for (int e = 0; e < 8; e++) {
        mag[e] = __float_as_uint(v[e]) & 0x7FFFFFFFu;
        lane_top = max(lane_top, mag[e]);
    }
    const uint32_t top = __reduce_max_sync(0xffffffffu, lane_top);
    w0 = 0u; w1 = 0u; s8 = 0; d = 0.0f;
    if (top == 0u) return;
    // First occurrence: the lowest lane that holds the maximum (ballot + find-first-set), its lowest such element.
    float lead = 0.0f;
    bool have = false;
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const bool hit = !have && mag[e] == top;
        lead = hit ? v[e] : lead;
        have = have || hit;
    }
    const int owner = __ffs((int)__ballot_sync(0xffffffffu, have)) - 1;
    const float iscale = __fdiv_rn(-127.0f, __shfl_sync(0xffffffffu, lead, owner));
    int qv[8];
#pragma unroll
    for (int e = 0; e < 8; e++) qv[e] = __float2int_rn(__fmul_rn(iscale, v[e]));   // >= -127; the pack clamps at +127
    w0 = pack_s8x4(qv[0], qv[1], qv[2], qv[3]);
    w1 = pack_s8x4(qv[4], qv[5], qv[6], qv[7]);
    s8 = __dp4a((int)w0, 0x01010101, __dp4a((int)w1, 0x01010101, 0));
    d = __fdiv_rn(1.0f, iscale);
}

// The same for NB blocks at a time (no sums), where every CTA of a several-column matvec forms all its columns' blocks and
// instructions count: the two divisions of each block are made by one lane per block at the same time, and where the largest
// magnitude is in [2^-100, 2^100] a product is rounded by adding 1.5 x 2^23, whose low byte then is the int8 value (|iscale * x|
// <= 127 (1 + 2^-23) rounds to at most 127), instead of a conversion on the quarter-rate unit (a block's eight took it 64
// clocks).  All other blocks (zeros, tiny, huge, infinite, NaN) are converted, out of line.  Seven columns of 5120 in the
// prologue of the matvec: 10,300 -> 6,800 clocks from the columns' arrival to the first weight.  (One column has one block a warp:
// there the longer code costs more than it saves, 27B-shaped pass 3810 -> 3850 us.)
static __device__ __noinline__ uint2 q8k_convert(float4 a, float4 b, float iscale) {
    const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    int q[8];
#pragma unroll
    for (int e = 0; e < 8; e++) q[e] = __float2int_rn(__fmul_rn(iscale, x[e]));   // >= -127; the pack clamps at +127
    return make_uint2(pack_s8x4(q[0], q[1], q[2], q[3]), pack_s8x4(q[4], q[5], q[6], q[7]));
}
__device__ __forceinline__ float max3_nan(float a, float b, float c) {   // NaN if any is
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
template <int NB>
__device__ __forceinline__ void q8k_blocks_core(const float (&v)[NB][8], uint32_t (&w0)[NB], uint32_t (&w1)[NB], float (&d)[NB]) {
    const int lane = threadIdx.x & 31;
    float mine = 1.0f;            // the leading element of block `lane`
    uint32_t tops[NB];
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const float (&x)[8] = v[b];
        // Magnitudes compare like their bit patterns, so the block maximum is an integer maximum: one REDUX over the warp.
        const float lane_top = max3_nan(max3_nan(fabsf(x[0]), fabsf(x[1]), fabsf(x[2])), max3_nan(fabsf(x[3]), fabsf(x[4]), fabsf(x[5])), max3_nan(fabsf(x[6]), fabsf(x[7]), 0.0f));
        tops[b] = __reduce_max_sync(0xffffffffu, __float_as_uint(lane_top) & 0x7FFFFFFFu);
        // First occurrence: the lowest lane that holds the maximum (ballot + find-first-set), there its first such element
        const float top = __uint_as_float(tops[b]);
        float lead = top;
#pragma unroll
        for (int e = 7; e >= 0; e--) lead = fabsf(x[e]) == top ? x[e] : lead;
        const int owner = __ffs((int)__ballot_sync(0xffffffffu, lane_top == top)) - 1;
        lead = __shfl_sync(0xffffffffu, lead, owner & 31);
        if (lane == b) mine = lead;
    }
    const float my_iscale = __fdiv_rn(-127.0f, mine), my_d = __fdiv_rn(1.0f, my_iscale);
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const float iscale = __shfl_sync(0xffffffffu, my_iscale, b);
        d[b] = __shfl_sync(0xffffffffu, my_d, b);
        if (tops[b] - 0x0D800000u <= 0x71800000u - 0x0D800000u) {   // 2^-100 .. 2^100
            uint32_t u[8];
#pragma unroll
            for (int e = 0; e < 8; e++) u[e] = __float_as_uint(__fadd_rn(__fmul_rn(iscale, v[b][e]), 12582912.0f));
            w0[b] = prmt(prmt(u[0], u[1], 0x0040u), prmt(u[2], u[3], 0x0040u), 0x5410u);
            w1[b] = prmt(prmt(u[4], u[5], 0x0040u), prmt(u[6], u[7], 0x0040u), 0x5410u);
        } else if (tops[b] == 0u) {
            w0[b] = w1[b] = 0u;
            d[b] = 0.0f;
        } else {
            const uint2 w = q8k_convert(make_float4(v[b][0], v[b][1], v[b][2], v[b][3]), make_float4(v[b][4], v[b][5], v[b][6], v[b][7]), iscale);
            w0[b] = w.x;
            w1[b] = w.y;
        }
    }
}
// The block as ggml lays it out (float d | int8 qs[256] | int16 bsums[16], 292 bytes, 4-byte aligned) from the core's
// outputs: lane l owns qs[8l .. 8l+7]; a bsum covers 16 values, i.e. a pair of lanes.
__device__ __forceinline__ void q8k_block_from_regs(const float (&v)[8], uint8_t* blk) {
    const int lane = threadIdx.x & 31;
    uint32_t w0, w1;
    int s8;
    float d;
    q8k_block_core(v, w0, w1, s8, d);
    uint32_t* words = (uint32_t*)blk;
    words[1 + 2 * lane] = w0;
    words[2 + 2 * lane] = w1;
    const int pair_sum = s8 + __shfl_down_sync(0xffffffffu, s8, 1);
    int16_t* bsums = (int16_t*)(blk + 4 + 256);
    if (!(lane & 1)) bsums[lane >> 1] = (int16_t)pair_sum;
    if (lane == 0) words[0] = __float_as_uint(d);
}

constexpr int Q8K_BYTES = 292;   // float d | int8 qs[256] | int16 bsums[16]  (src/quant/quant_formats.h:95)
constexpr int ACT_WARPS = 8;

// One warp quantizes 256 floats at `src` (lane l holds elements 8l..8l+7) into the Q8_K block at `blk`.
// COHERENT: read through L2 only (the floats were written by another SM during this kernel).
template <bool COHERENT>
__device__ __forceinline__ void quantize_block(const float* src, uint8_t* blk) {
    const int lane = threadIdx.x & 31;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = COHERENT ? __ldcg(src + 8 * lane + e) : src[8 * lane + e];
    q8k_block_from_regs(v, blk);
}

// h = silu(g) * u, the CPU formula of the reference (src/runtime/engine.cpp:177-182): g / (1 + expf(-g)) * u
__device__ __forceinline__ float swiglu_value(float gv, float uv) { return __fmul_rn(__fdiv_rn(gv, __fadd_rn(1.0f, expf(-gv))), uv); }

// one warp, 256 values
template <bool COHERENT>
__device__ __forceinline__ void swiglu_block(const float* g, const float* u, float* h, uint8_t* blk) {
    const int lane = threadIdx.x & 31;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const float gv = COHERENT ? __ldcg(g + 8 * lane + e) : g[8 * lane + e];
        const float uv = COHERENT ? __ldcg(u + 8 * lane + e) : u[8 * lane + e];
        v[e] = swiglu_value(gv, uv);
    }
    if (h) {
#pragma unroll
        for (int e = 0; e < 8; e++) h[8 * lane + e] = v[e];
    }
    if (blk) q8k_block_from_regs(v, blk);
}

static __global__ void __launch_bounds__(ACT_WARPS * 32) quantize_q8k_kernel(const float* __restrict__ x, long long x_ld, int K,
                                                                       int n_rows, uint8_t* __restrict__ out,
                                                                       long long out_stride) {
    const int nsb = K >> 8;
    const long long blk = (long long)blockIdx.x * ACT_WARPS + (threadIdx.x >> 5);
    if (blk >= (long long)n_rows * nsb) return;
    const int r = (int)(blk / nsb), sb = (int)(blk % nsb);
    quantize_block<false>(x + (size_t)r * x_ld + (size_t)sb * 256, out + ((size_t)r * out_stride + sb) * 292);
}

// The reference GPU path's activation format (ActQ8, src/cuda/gemv.cuh:14-21; quantizer src/cuda/gemv.cu:31-47): one
// warp per 32 values, d = amax / 127, q = round-half-even(v / d) (an all-zero block stays zero), s = d * sum q.
static __global__ void __launch_bounds__(ACT_WARPS * 32) quantize_act_q8_kernel(const float* __restrict__ x, long long n_blocks,
                                                                          int8_t* __restrict__ q, float* __restrict__ d,
                                                                          float* __restrict__ s) {
    const long long blk = (long long)blockIdx.x * ACT_WARPS + (threadIdx.x >> 5);
    if (blk >= n_blocks) return;
    const int lane = threadIdx.x & 31;
    const float v = x[blk * 32 + lane];
    const float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v) & 0x7FFFFFFFu));
    const float dd = __fdiv_rn(amax, 127.0f);
    const int qi = dd > 0.0f ? __float2int_rn(__fdiv_rn(v, dd)) : 0;
    q[blk * 32 + lane] = (int8_t)qi;
    const int sum = __reduce_add_sync(0xffffffffu, qi);
    if (lane == 0) {
        d[blk] = dd;
        s[blk] = __fmul_rn(dd, (float)sum);
    }
}

static __global__ void __launch_bounds__(ACT_WARPS * 32) swiglu_q8k_kernel(const float* __restrict__ g, const float* __restrict__ u,
                                                                     long long ld, int n, int n_rows, float* __restrict__ h,
                                                                     uint8_t* __restrict__ out, long long out_stride,
                                                                     const PeerSync sync, int* status) {
    if (sync.n > 0) {   // gate and up were completed by the other GPUs: cross-GPU barrier first
        peer_sync_wait(sync, blockIdx.x == 0, (int)threadIdx.x, status);
        __syncthreads();
    }
    const int nsb = n >> 8;
    const long long blk = (long long)blockIdx.x * ACT_WARPS + (threadIdx.x >> 5);
    if (blk >= (long long)n_rows * nsb) return;
    const int r = (int)(blk / nsb), sb = (int)(blk % nsb);
    const size_t off = (size_t)r * ld + (size_t)sb * 256;
    swiglu_block<false>(g + off, u + off, h ? h + off : nullptr, out ? out + ((size_t)r * out_stride + sb) * 292 : nullptr);
}

// Residual add + RMSNorm + Q8_K in one pass over the row (replaces k_add_rmsnorm feeding the matvecs,
// src/cuda/ops.cu:78-123): x += a (+ b) is written back (the residual stream), xn = x * rsqrt(mean(x^2) + eps) * w goes
// out as fp32 (optional) and as the Q8_K blocks the next matvecs read.  One CTA per row, one warp per 256 values: every
// value stays in a register from the load to the quantizer.  n a multiple of 256, at most 32 * 256.
static __global__ void __launch_bounds__(1024) add_rmsnorm_q8k_kernel(float* __restrict__ x, const float* __restrict__ a,
                                                                      const float* __restrict__ b, const float* __restrict__ w, int n,
                                                                      long long ld, float eps, float* __restrict__ xn,
                                                                      uint8_t* __restrict__ q8k, long long q8k_stride) {
    __shared__ float part[32];
    __shared__ float s_scale;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const size_t ro = (size_t)blockIdx.x * ld, at = ro + (size_t)warp * 256 + 8 * lane;
    float v[8];
    {
        const float4 lo = *(const float4*)(x + at), hi = *(const float4*)(x + at + 4);
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    }
    if (a) {
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = __fadd_rn(v[e], a[at + e]);
    }
    if (b) {
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = __fadd_rn(v[e], b[at + e]);
    }
    if (a || b) {
        *(float4*)(x + at) = make_float4(v[0], v[1], v[2], v[3]);
        *(float4*)(x + at + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
    float ss = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; e++) ss = fmaf(v[e], v[e], ss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nw ? part[lane] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) s_scale = rsqrtf(t / (float)n + eps);
    }
    __syncthreads();
    const float scale = s_scale;
    const float4 wl = *(const float4*)(w + (size_t)warp * 256 + 8 * lane), wh = *(const float4*)(w + (size_t)warp * 256 + 8 * lane + 4);
    const float ww[8] = {wl.x, wl.y, wl.z, wl.w, wh.x, wh.y, wh.z, wh.w};
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = __fmul_rn(__fmul_rn(v[e], scale), ww[e]);
    if (xn) {
        *(float4*)(xn + at) = make_float4(v[0], v[1], v[2], v[3]);
        *(float4*)(xn + at + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
    if (q8k) q8k_block_from_regs(v, q8k + ((size_t)blockIdx.x * q8k_stride + warp) * 292);
}

// y[r] = W[r,:] . x for dense bf16 weights (the model's two small per-layer projections, 48 x 5120; replaces gemv_bf16,
// src/cuda/gemv.cu:127-146, 235-238).  One CTA of BF16_THREADS per row: every thread takes 16-byte pieces (eight bf16) of
// the row, fp32 multiply-adds, a shuffle tree per warp and a last add over the warps in shared memory.
constexpr int BF16_THREADS = 128;
static __global__ void __launch_bounds__(BF16_THREADS) gemv_bf16_kernel(const uint16_t* __restrict__ W, int K, int N,
                                                                       const float* __restrict__ x, float* __restrict__ y) {
    __shared__ float part[BF16_THREADS / 32];
    const int row = blockIdx.x, tid = threadIdx.x;
    const uint4* w = (const uint4*)(W + (size_t)row * K);
    float acc = 0.0f;
    for (int i = tid; i < K / 8; i += BF16_THREADS) {
        const uint4 p = w[i];
        const float4 xa = *(const float4*)(x + 8 * i), xb = *(const float4*)(x + 8 * i + 4);
        // a bf16 is the upper half of an fp32
        acc = fmaf(__uint_as_float(p.x << 16), xa.x, acc); acc = fmaf(__uint_as_float(p.x & 0xFFFF0000u), xa.y, acc);
        acc = fmaf(__uint_as_float(p.y << 16), xa.z, acc); acc = fmaf(__uint_as_float(p.y & 0xFFFF0000u), xa.w, acc);
        acc = fmaf(__uint_as_float(p.z << 16), xb.x, acc); acc = fmaf(__uint_as_float(p.z & 0xFFFF0000u), xb.y, acc);
        acc = fmaf(__uint_as_float(p.w << 16), xb.z, acc); acc = fmaf(__uint_as_float(p.w & 0xFFFF0000u), xb.w, acc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((tid & 31) == 0) part[tid >> 5] = acc;
    __syncthreads();
    if (tid == 0) {
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < BF16_THREADS / 32; i++) s += part[i];
        y[row] = s;
    }
}

// Prefill SwiGLU in place (replaces swiglu_rows_inplace, src/cuda/prefill.cu:132-151): row b of silu(G) * U, n values,
// overwrites the first 2 n bytes of G's row b as 16-bit floats (fp16 like the reference, or bf16 for the bf16 GEMM).
// One CTA per row: the whole result row is formed in shared memory first (2 n bytes), then copied over the row's start,
// so no read of G can see a half written earlier.  n, ld multiples of 8; 2 n bytes of shared memory.
// Bound by memory (10 bytes a value): 512 threads with four 16-byte loads each in flight; with 256 threads and 8-byte loads
// 1024 x 17408 took 56 us, now 35 us (5.1 TB/s).  Rows of less than 2048 values take fewer threads (512 threads leave warps
// with nothing to load: 2500 x 512 8.6 us, with 128 threads 4.6 us; 2500 x 1024 10.5 and, with 256, 7.7 us).
inline int swiglu_rows_threads(int n) { return n >= 2048 ? 512 : n >= 1024 ? 256 : 128; }
template <bool BF16, int SWIGLU_ROWS_THREADS>
static __global__ void __launch_bounds__(SWIGLU_ROWS_THREADS, 1536 / SWIGLU_ROWS_THREADS) swiglu_rows_inplace_kernel(float* G, const float* __restrict__ U, int n, long long ld) {
    extern __shared__ __align__(16) uint8_t row_smem[];
    float* g = G + (size_t)blockIdx.x * ld;
    const float* u = U + (size_t)blockIdx.x * ld;
    auto value = [](float x, float y) { return x / (1.0f + __expf(-x)) * y; };
    auto pack = [](float x, float y) {
        uint32_t w;
        if (BF16) { const __nv_bfloat162 v = __floats2bfloat162_rn(x, y); w = *(const uint32_t*)&v; }
        else { const __half2 v = __floats2half2_rn(x, y); w = *(const uint32_t*)&v; }
        return w;
    };
    const int n4 = n / 4;
    for (int i0 = threadIdx.x; i0 < n4; i0 += 2 * SWIGLU_ROWS_THREADS) {
        const int i1 = i0 + SWIGLU_ROWS_THREADS;
        const bool two = i1 < n4;
        const float4 a0 = ((const float4*)g)[i0], b0 = ((const float4*)u)[i0];
        float4 a1 = make_float4(0.f, 0.f, 0.f, 0.f), b1 = a1;
        if (two) { a1 = ((const float4*)g)[i1]; b1 = ((const float4*)u)[i1]; }
        ((uint2*)row_smem)[i0] = make_uint2(pack(value(a0.x, b0.x), value(a0.y, b0.y)), pack(value(a0.z, b0.z), value(a0.w, b0.w)));
        if (two) ((uint2*)row_smem)[i1] = make_uint2(pack(value(a1.x, b1.x), value(a1.y, b1.y)), pack(value(a1.z, b1.z), value(a1.w, b1.w)));
    }
    __syncthreads();
    uint4* dst = (uint4*)g;
    const uint4* src = (const uint4*)row_smem;
    for (int i = threadIdx.x; i < n / 8; i += SWIGLU_ROWS_THREADS) dst[i] = src[i];
}

}  // namespace q38b
