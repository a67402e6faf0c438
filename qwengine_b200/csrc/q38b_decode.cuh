// q38b_decode.cuh -- per-format tensor-core fragment builders of the several-column matvec.
//
// One warp multiplies 16 rows of a GGUF weight matrix (staged in shared memory in their file layout) with up to 8 int8
// activation columns, a 256-weight super-block at a time.  Lane (g = lane / 4, t = lane % 4) decodes weights of rows g and
// g + 8 straight into the A fragments of mma.sync.m16n8k32.s8 (m16n8k16 where the scale changes every 16 weights); the
// activations are the B fragments.  Each mma yields exact int32 dot products, which are multiplied by the integer
// sub-block scale and summed in int32 over the whole super-block; then d_weight * d_activation is applied once.
// These are the same exact integer sums as the reference CPU kernels form
// (src/cpu/cpu_kernels.cpp:130-515 of the reference project), so results differ from them only by
// the order of the float additions.
//
// The order of the 32 k-slots of one mma is free as long as A and B agree.  Every format maps lane
// t to the 8 weights that its own bytes hold:
//   IQ3_XXS, IQ3_S, Q4_K, Q5_K, Q8_0, IQ2_*, IQ1_*: weights 8t..8t+7 of the sub-block (B = 8 consecutive int8);
//   IQ4_XS: weights 4t..4t+3 and 16+4t..19+4t interleaved (activations are staged in that order);
//   Q6_K, Q2_K: weights 4t..4t+3 of each 16-weight group (k16 mma).
// Columns g >= nb carry column 0's values: their sums are never stored, so no lane zeroes its fragment.
//
// What bounds these decoders is the number of instructions per weight (the tensor pipe is a few percent busy, HBM waits):
// everything that belongs to a row's super-block (scale bytes, sign words) is loaded and unpacked once per super-block
// (Row), words that all four lanes of a row need are loaded by one of them and shuffled, the products with negative
// weights are a second mma on masked magnitudes instead of byte-wise negations where that saves arithmetic.
//
// The file compiles for the device and, with the warp-collective operations replaced by an
// emulation that the CPU unit test provides, for the host.
#pragma once
#include <cstdint>
#include <cstring>
#include <cmath>
#if !defined(__CUDA_ARCH__)
#include <cstdio>
#include <cstdlib>
#endif

#if defined(__CUDACC__)
#include <cuda_fp16.h>
#define Q38B_HD __host__ __device__ __forceinline__
#else
#define Q38B_HD inline
#endif

namespace q38b {

// ggml type ids (the reference keeps them verbatim: include/q38rt/q38rt_types.h:36-67)
enum : int { T_Q8_0 = 8, T_Q4_K = 12, T_Q5_K = 13, T_Q6_K = 14, T_IQ3_XXS = 18, T_IQ3_S = 21, T_IQ4_XS = 23,
              // the reference has these too:
              T_Q2_K = 10, T_IQ2_XXS = 16, T_IQ2_XS = 17, T_IQ1_S = 19, T_IQ2_S = 22, T_IQ1_M = 29 };

#if !defined(__CUDA_ARCH__)
// Host emulation hooks (defined by the CPU unit test): current lane, warp-wide mma and shuffle.
int emul_lane();
void emul_mma(int (&c)[4], const uint32_t* a, int n_a, const uint32_t* b, int n_b);
uint32_t emul_shfl(uint32_t v, int src_lane);
#endif

// ------------------------------------------------------------------------------------------------
// Scalar helpers
// ------------------------------------------------------------------------------------------------
Q38B_HD int lane_id() {
#if defined(__CUDA_ARCH__)
    return (int)(threadIdx.x & 31u);
#else
    return emul_lane();
#endif
}

// PRMT: byte i of the result = byte (sel nibble i & 7) of {a (bytes 0-3), b (bytes 4-7)}; nibble bit 3 set
// replicates that byte's sign bit instead.
Q38B_HD uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
#if defined(__CUDA_ARCH__)
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
#else
    const uint64_t v = (uint64_t)a | ((uint64_t)b << 32);
    uint32_t r = 0;
    for (int i = 0; i < 4; i++) {
        const uint32_t n = (sel >> (4 * i)) & 0xF;
        uint32_t byte = (uint32_t)(v >> (8 * (n & 7))) & 0xFF;
        if (n & 8) byte = (byte & 0x80) ? 0xFF : 0x00;
        r |= byte << (8 * i);
    }
    return r;
#endif
}

Q38B_HD int popc(uint32_t v) {
#if defined(__CUDA_ARCH__)
    return __popc(v);
#else
    return __builtin_popcount(v);
#endif
}

Q38B_HD float fp16_bits_to_float(uint32_t h) {
#if defined(__CUDA_ARCH__)
    return __half2float(__ushort_as_half((unsigned short)h));   // exact, subnormals included
#else
    const uint32_t sign = (h & 0x8000u) << 16;
    int exp = (h >> 10) & 0x1F;
    uint32_t mant = h & 0x3FFu, bits;
    if (exp == 0) {
        if (!mant) bits = sign;
        else { int e = 113; while (!(mant & 0x400u)) { mant <<= 1; e--; } bits = sign | ((uint32_t)e << 23) | ((mant & 0x3FFu) << 13); }
    } else if (exp == 31) bits = sign | 0x7F800000u | (mant << 13);
    else bits = sign | ((uint32_t)(exp + 112) << 23) | (mant << 13);
    float f; memcpy(&f, &bits, 4); return f;
#endif
}

Q38B_HD uint32_t funnel_r(uint32_t lo, uint32_t hi, uint32_t sh) {   // (hi:lo) >> sh, sh in 0..31
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, sh);
#else
    return sh ? (lo >> sh) | (hi << (32 - sh)) : lo;
#endif
}

// ---------------------------------------------------------------------------------------------------------------
// Staged bytes are addressed through SP: on the device a 32-bit shared-space address (loads are ld.shared with
// immediate offsets, no 64-bit pointer arithmetic and no generic-to-shared conversion per load), on the host a pointer.
// ---------------------------------------------------------------------------------------------------------------
#if defined(__CUDA_ARCH__)
struct SP { uint32_t a; };
__device__ __forceinline__ SP sp_from(const void* p) { return SP{(uint32_t)__cvta_generic_to_shared(p)}; }
__device__ __forceinline__ uint32_t sp_low2(SP p) { return p.a & 2u; }
__device__ __forceinline__ uint32_t sp_ld8(SP p, int o = 0) { uint32_t v; asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(p.a + o)); return v; }
__device__ __forceinline__ int sp_ld8s(SP p, int o = 0) { int v; asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(p.a + o)); return v; }
__device__ __forceinline__ uint32_t sp_ld16(SP p, int o = 0) { uint32_t v; asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(p.a + o)); return v; }
__device__ __forceinline__ uint32_t sp_ld32(SP p, int o = 0) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p.a + o)); return v; }
__device__ __forceinline__ float sp_ldf(SP p, int o = 0) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p.a + o)); return v; }
__device__ __forceinline__ void sp_ld64(SP p, int o, uint32_t& x, uint32_t& y) {
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(x), "=r"(y) : "r"(p.a + o));
}
__device__ __forceinline__ void sp_ld128(SP p, int o, uint32_t (&v)[4]) {
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(p.a + o));
}
#else
struct SP { const uint8_t* a; };
inline SP sp_from(const void* p) { return SP{(const uint8_t*)p}; }
inline uint32_t sp_low2(SP p) { return (uint32_t)((uintptr_t)p.a & 2); }
inline uint32_t sp_ld8(SP p, int o = 0) { return p.a[o]; }
inline int sp_ld8s(SP p, int o = 0) { return (int8_t)p.a[o]; }
// the host versions refuse what the device would fault on: an address that is not a multiple of the access size
inline void sp_check_aligned(const uint8_t* p, int n) { if ((uintptr_t)p % (uintptr_t)n) { fprintf(stderr, "misaligned %d-byte shared load\n", n); abort(); } }
inline uint32_t sp_ld16(SP p, int o = 0) { uint16_t v; sp_check_aligned(p.a + o, 2); memcpy(&v, p.a + o, 2); return v; }
inline uint32_t sp_ld32(SP p, int o = 0) { uint32_t v; sp_check_aligned(p.a + o, 4); memcpy(&v, p.a + o, 4); return v; }
inline float sp_ldf(SP p, int o = 0) { float v; sp_check_aligned(p.a + o, 4); memcpy(&v, p.a + o, 4); return v; }
inline void sp_ld64(SP p, int o, uint32_t& x, uint32_t& y) { sp_check_aligned(p.a + o, 8); memcpy(&x, p.a + o, 4); memcpy(&y, p.a + o + 4, 4); }
inline void sp_ld128(SP p, int o, uint32_t (&v)[4]) { sp_check_aligned(p.a + o, 16); memcpy(v, p.a + o, 16); }
#endif
Q38B_HD SP operator+(SP p, int o) { return SP{p.a + o}; }
Q38B_HD SP operator-(SP p, int o) { return SP{p.a - o}; }

// 8 bytes from a 2-byte aligned address: three aligned words and two funnel shifts.  `mis` = address & 2.
Q38B_HD void sp_ld8b_a2(SP p, uint32_t mis, uint32_t& lo, uint32_t& hi) {
    const SP w = p - (int)mis;
    const uint32_t sh = mis * 8;
    const uint32_t w0 = sp_ld32(w, 0), w1 = sp_ld32(w, 4), w2 = sp_ld32(w, 8);
    lo = funnel_r(w0, w1, sh);
    hi = funnel_r(w1, w2, sh);
}

// D(16x8,s32) = A(16x32,s8) * B(32x8,s8) + C.  Fragment layout of PTX mma.m16n8k32 (g = lane/4, t = lane%4):
// a0 = A[g][4t..4t+3], a1 = A[g+8][4t..], a2 = A[g][16+4t..], a3 = A[g+8][16+4t..]; b0 = B[4t..4t+3][g],
// b1 = B[16+4t..][g]; c0,c1 = C[g][2t,2t+1], c2,c3 = C[g+8][2t,2t+1].
Q38B_HD void mma_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
#if defined(__CUDA_ARCH__)
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
#else
    const uint32_t a[4] = {a0, a1, a2, a3}, b[2] = {b0, b1};
    emul_mma(c, a, 4, b, 2);
#endif
}
// C = 0
Q38B_HD void mma_k32_z(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
#if defined(__CUDA_ARCH__)
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
#else
    c[0] = c[1] = c[2] = c[3] = 0;
    mma_k32(c, a0, a1, a2, a3, b0, b1);
#endif
}
// k16 variant: a0 = A[g][4t..4t+3], a1 = A[g+8][4t..]; b0 = B[4t..4t+3][g].
Q38B_HD void mma_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
#if defined(__CUDA_ARCH__)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0));
#else
    const uint32_t a[2] = {a0, a1}, b[1] = {b0};
    emul_mma(c, a, 2, b, 1);
#endif
}
Q38B_HD void mma_k16_z(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
#if defined(__CUDA_ARCH__)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(0));
#else
    c[0] = c[1] = c[2] = c[3] = 0;
    mma_k16(c, a0, a1, b0);
#endif
}

// the value of lane `j` of this lane's group of four
Q38B_HD uint32_t quad_shfl(uint32_t v, int j) {
#if defined(__CUDA_ARCH__)
    return __shfl_sync(0xffffffffu, v, j, 4);
#else
    return emul_shfl(v, (emul_lane() & ~3) | j);
#endif
}

// Byte mask (0xFF where the sign bit is set) for 4 weights from a 4-bit field: one multiply moves
// bit i to the top bit of byte i (the shifted copies never overlap, so no carries), PRMT's
// sign-replicate mode widens each top bit to a whole byte.  `nib` may carry garbage in bits 4..6.
Q38B_HD uint32_t sign_mask4(uint32_t nib) { return prmt(nib * 0x10204080u, 0u, 0xBA98u); }

// Negate the bytes of g selected by mask m (0xFF / 0x00 per byte).  Codebook magnitudes are never 0,
// so (g ^ 0xFF) + 1 = 256 - g stays inside its byte.
Q38B_HD uint32_t negate_bytes(uint32_t g, uint32_t m) { return (g ^ m) + (m & 0x01010101u); }

// Activation operand of one lane for one super-block (the CPU unit test's interface to the fragment builders).
struct ActLane {
    const uint8_t* q;   // int8 activations of column g for this super-block (256 bytes, staged order); column 0's where !valid
    bool valid;         // column g < nb (for the test's own use: the fragments multiply column 0 there)
    float dx0, dx1;     // Q8_K block scales of columns 2t and 2t+1 (0 beyond nb)
};

// Codebook in shared memory, replicated so that lane l reads bank l: entry e, replica r at
// word (e << rep_log2) + r, r = lane & (2^rep_log2 - 1).
struct Codebook {
    const uint32_t* words;
    int rep_log2;
    uint32_t lane_word;   // lane & (replicas - 1)
};

// What a warp's lane works with: the staged activations of its column, its tables.
//   q        column g, this super-block, 8 t bytes in (4 t for the k16 formats)
//   q_half   the same where the lane's weights belong to half h of the sub-block, else a run of zeros (formats whose scale
//            changes every 16 weights but whose grid entries are eight: lanes 0, 1 hold the first half, 2, 3 the second)
//   cb       32-bit codebook: entry e at cb + (e << cb_shift); grid8: eight-byte grid entries likewise
//   sgn      byte masks of the 128 seven-bit sign codes, SIGN_COPIES times: code c at sgn + 8 c SIGN_COPIES (TABLES; else they
//            are computed, with seven operations where the look-up takes two)
//   bsum     this lane's word of the staged sums of activations (TABLES; see the minima below)
constexpr int SIGN_COPIES = 8, SIGN_STRIDE_LOG2 = 6;   // (16 would meet no bank but cost the ring 8 KB)
struct FragEnv {
    SP q, q_half[2];
    SP cb, sgn, bsum;
    int cb_shift;
    int t;
};
// The minima of the K-quants: sum over the sub-blocks of m * (sum of the sub-block's activations).  TABLES: the sums are
// staged as two digits, 64 hi + lo, and one k16 mma per digit and super-block forms the product (per column 8 lo | 8 hi bytes
// a super-block, Q2_K 16 lo | 16 hi); else m is broadcast to every slot of a second mma per sub-block (per-32 activations,
// whose scales differ by sub-block; the unit test).  Eight IMMA a super-block less: Q4_K's decoder 334 -> 275 clocks
// per warp and super-block (an IMMA keeps the issue port of the integer units busy for nine clocks).

Q38B_HD uint32_t ld_u32_a2(SP p, int o) { return prmt(sp_ld16(p, o), sp_ld16(p, o + 2), 0x5410u); }
// byte k of w, zero or sign extended
Q38B_HD int byte_u(uint32_t w, int k) { return (int)prmt(w, 0u, 0x4440u | (uint32_t)k); }
Q38B_HD int byte_s(uint32_t w, int k) { return (int)prmt(w, 0u, (uint32_t)(k | ((8 | k) << 4) | ((8 | k) << 8) | ((8 | k) << 12))); }

// Sign masks of eight weights from seven sign bits, the eighth their parity
Q38B_HD void sign_masks7(uint32_t s7, uint32_t& lo, uint32_t& hi) {
    lo = sign_mask4(s7);
    hi = prmt((uint32_t)popc(s7) * 0x80000000u + s7 * 0x00020408u, 0u, 0xBA98u);
}
// ... of the bits [at, at + 7) of w, by look-up (a shift, a mask and a load that is served in two to three wavefronts) or computed
// (seven operations).  The decoders look up row g's masks and compute row g + 8's: all by look-up the shared-memory pipe
// sets the pace (2 x 17408 x 5120 IQ3_XXS, seven columns: 40.1 us), all computed the integer units (38.4 us), half and half 37.5.
template <bool TABLES>
Q38B_HD void sign_masks7_at(const FragEnv& e, uint32_t w, int at, uint32_t& lo, uint32_t& hi) {   // bits [at, at + 7) of w
    if constexpr (TABLES) {
        // rotated so that the field starts at the bit of the entry's stride
        sp_ld64(e.sgn + (int)(funnel_r(w, w, (uint32_t)(at + 32 - SIGN_STRIDE_LOG2) & 31u) & (127u << SIGN_STRIDE_LOG2)), 0, lo, hi);
    } else {
        sign_masks7((w >> at) & 127u, lo, hi);
    }
}
// ... from eight sign bits
Q38B_HD void sign_masks8(uint32_t s8, uint32_t& lo, uint32_t& hi) {
    lo = sign_mask4(s8 & 0x7Fu);
    hi = sign_mask4(s8 >> 4);
}

// d_weight * d_activation * (integer sum of a super-block), less d_min * d_activation * (integer sum of the minima): written
// out so that the one-column and the several-column kernels round alike whatever the compiler would contract
Q38B_HD float fmul_once(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
Q38B_HD float block_value(float ddx, int sum) { return fmul_once(ddx, (float)sum); }
Q38B_HD float block_value_min(float ddx, int sum, float mdx, int msum) { return fmaf(-mdx, (float)msum, fmul_once(ddx, (float)sum)); }

// Unit<FMT>: Row = what is loaded once per row and super-block; half() = 128 weights of 16 rows, calling emit(s, v) for each
// of its four 32-weight sub-blocks s with v[i] = sum of scale * weight * activation (i as in mma's C: rows g, g, g + 8, g + 8;
// columns 2t, 2t + 1, ...) and adding the minimum's part to cm; dd() = the row's float factors.
//   FACTOR   a power of two every value carries (0.25 for the IQ3_XXS scale (2s + 1) / 4, ...)
//   HAS_MIN  minima (Q4_K, Q5_K, Q2_K)
// half<TABLES>: sign masks by look-up, minima by mins() from the staged sums.
template <int FMT> struct Unit;

// the common tail of the unit test's interface: one half super-block with Q8_K activations
template <int FMT>
Q38B_HD void unit_run(const uint8_t* pA8, const uint8_t* pB8, int h, const ActLane& act, const Codebook& cb, float (&acc)[4]) {
    using U = Unit<FMT>;
    const SP pA = sp_from(pA8), pB = sp_from(pB8);
    FragEnv e;
    e.t = lane_id() & 3;
    e.q = sp_from(act.q) + U::ACT_STEP * e.t;
    e.q_half[0] = e.q_half[1] = e.q;
    e.cb = sp_from((const uint8_t*)(cb.words + cb.lane_word));
    e.cb_shift = cb.rep_log2 + 2;
    typename U::Row A, B;
    U::row(pA, e.t, A);
    U::row(pB, e.t, B);
    int sumi[4] = {0, 0, 0, 0}, cm[4] = {0, 0, 0, 0};
    float d32[4] = {0.f, 0.f, 0.f, 0.f};
    U::template half<false>(A, B, pA, pB, h, e, cm, [&](int s, const int (&v)[4]) {
        for (int i = 0; i < 4; i++) {
            if (U::SCALE32) d32[i] += block_value(U::d32(i < 2 ? pA : pB, s), v[i]);
            else sumi[i] += v[i];
        }
    });
    float dA, mA, dB, mB;
    U::dd(pA, A, dA, mA);
    U::dd(pB, B, dB, mB);
    for (int i = 0; i < 4; i++) {
        const float dx = (i & 1) ? act.dx1 : act.dx0, d = i < 2 ? dA : dB, m = i < 2 ? mA : mB;
        acc[i] += U::SCALE32 ? d32[i] * dx : U::HAS_MIN ? block_value_min(d * dx, sumi[i], m * dx, cm[i]) : block_value(d * dx * U::FACTOR, sumi[i]);
    }
}
template <int FMT> struct UnitRun {
    static constexpr int ACT_STEP = 8;           // bytes of a sub-block between the lanes t of a row
    static constexpr bool SCALE32 = false, HAS_MIN = false;
    static constexpr float FACTOR = 1.0f;
    static Q38B_HD float d32(SP, int) { return 0.0f; }
    static Q38B_HD void run(const uint8_t* pA, const uint8_t* pB, int h, const ActLane& act, const Codebook& cb, float (&acc)[4]) {
        unit_run<FMT>(pA, pB, h, act, cb, acc);
    }
};

// Position inside a 32-activation sub-block at which activation k is staged for a format.
Q38B_HD int act_stage_pos(int fmt, int k) {
    if (fmt != T_IQ4_XS) return k;
    // lane t holds qs bytes 4t..4t+3; nibbles in selector order: (4t, 16+4t, 4t+1, 17+4t | 4t+2, 18+4t, 4t+3, 19+4t)
    const int hi = k >> 4, r = k & 15, t = r >> 2, i = r & 3;
    return 8 * t + 2 * i + hi;
}

// Weights given as magnitudes g and sign masks m (0xFF where negative), rows A and B: one mma on the magnitudes, one on those
// of the negative weights, v = scale * (c - 2 n).  Four ANDs and four multiply-adds per 16 weights where negating the bytes takes twelve operations.
struct Signed8 { uint32_t g0, g1, m0, m1; };
Q38B_HD void mma_signed(const Signed8& A, const Signed8& B, uint32_t b0, uint32_t b1, int scA, int scB, int (&v)[4]) {
    int c[4], n[4];
    mma_k32_z(c, A.g0, B.g0, A.g1, B.g1, b0, b1);
    mma_k32_z(n, A.g0 & A.m0, B.g0 & B.m0, A.g1 & A.m1, B.g1 & B.m1, b0, b1);
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = (i < 2 ? scA : scB) * (c[i] - 2 * n[i]);
}

// ------------------------------------------------------------------------------------------------
// IQ3_XXS: 98 bytes = fp16 d | 64 grid indices | 8 x u32 (4 x 7 sign-index bits + 4-bit scale).
// w = d * (0.5 + s) * 0.5 * grid * sign (src/quant/quant_ref.cpp:165-188); integer form
// sum (2s+1) * grid * sign * q8, scaled by d * dx * 0.25 (src/cpu/cpu_kernels.cpp:164-189).
// Lane t loads the sign / scale words of sub-blocks t and t + 4 and hands them to the row's other lanes.
// ------------------------------------------------------------------------------------------------
template <> struct Unit<T_IQ3_XXS> : UnitRun<T_IQ3_XXS> {
    static constexpr int BLOCK_BYTES = 98;
    static constexpr int CODEBOOK_ENTRIES = 256;
    static constexpr float FACTOR = 0.25f;
    struct Row { uint32_t aux[2]; };

    static Q38B_HD void row(SP p, int t, Row& r) {
        r.aux[0] = ld_u32_a2(p + 4 * t, 66);
        r.aux[1] = ld_u32_a2(p + 4 * t, 82);
    }
    static Q38B_HD void dd(SP p, const Row&, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(p, 0)); m = 0.0f; }
    template <bool TABLES>
    static Q38B_HD void weights(SP p2t, int s, uint32_t aux, const FragEnv& e, Signed8& w, int& scale) {
        const uint32_t idx = sp_ld16(p2t, 2 + 8 * s);
        w.g0 = sp_ld32(e.cb + (int)((idx & 0xFFu) << e.cb_shift));
        w.g1 = sp_ld32(e.cb + (int)((idx >> 8) << e.cb_shift));
        sign_masks7_at<TABLES>(e, aux, 7 * e.t, w.m0, w.m1);
        scale = (int)(2u * (aux >> 28) + 1u);
    }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA2 = pA + 2 * e.t, pB2 = pB + 2 * e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            Signed8 wA, wB;
            int scA, scB, v[4];
            weights<TABLES>(pA2, s, quad_shfl(A.aux[h], j), e, wA, scA);
            weights<false>(pB2, s, quad_shfl(B.aux[h], j), e, wB, scB);
            uint32_t b0, b1;
            sp_ld64(e.q, 32 * s, b0, b1);
            mma_signed(wA, wB, b0, b1, scA, scB, v);
            emit(s, v);
        }
    }
};

// ------------------------------------------------------------------------------------------------
// IQ3_S: 110 bytes = fp16 d | qs[64] | qh[8] (9th index bits) | signs[32] | scales[4] (nibbles).
// w = d * (1 + 2 ls) * grid * sign (src/quant/quant_ref.cpp:190-225; src/cpu/cpu_kernels.cpp:130-162).
// ------------------------------------------------------------------------------------------------
template <> struct Unit<T_IQ3_S> : UnitRun<T_IQ3_S> {
    static constexpr int BLOCK_BYTES = 110;
    static constexpr int CODEBOOK_ENTRIES = 512;
    struct Row { uint32_t qh[2], sc; };   // qh: the ninth index bits of sub-blocks 0..3 / 4..7, shifted so that this lane's two are bits 8 j, 8 j + 1

    static Q38B_HD void row(SP p, int t, Row& r) {
        r.qh[0] = ld_u32_a2(p, 66) >> (2 * t);
        r.qh[1] = ld_u32_a2(p, 70) >> (2 * t);
        r.sc = ld_u32_a2(p, 106);
    }
    static Q38B_HD void dd(SP p, const Row&, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(p, 0)); m = 0.0f; }
    static Q38B_HD void weights(const Row& r, SP p2t, SP pt, int s, const FragEnv& e, Signed8& w, int& scale) {
        const uint32_t idx = sp_ld16(p2t, 2 + 8 * s), hb = r.qh[s >> 2] >> (8 * (s & 3));
        w.g0 = sp_ld32(e.cb + (int)(((idx & 0xFFu) | ((hb & 1u) << 8)) << e.cb_shift));
        w.g1 = sp_ld32(e.cb + (int)(((idx >> 8) | ((hb & 2u) << 7)) << e.cb_shift));
        sign_masks8(sp_ld8(pt, 74 + 4 * s), w.m0, w.m1);
        scale = (int)((s == 0 ? (r.sc << 1) : (r.sc >> (4 * s - 1))) & 0x1Eu) + 1;
    }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA1 = pA + e.t, pB1 = pB + e.t, pA2 = pA1 + e.t, pB2 = pB1 + e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            Signed8 wA, wB;
            int scA, scB, v[4];
            weights(A, pA2, pA1, s, e, wA, scA);
            weights(B, pB2, pB1, s, e, wB, scB);
            uint32_t b0, b1;
            sp_ld64(e.q, 32 * s, b0, b1);
            mma_signed(wA, wB, b0, b1, scA, scB, v);
            emit(s, v);
        }
    }
};

// ------------------------------------------------------------------------------------------------
// IQ4_XS: 136 bytes = fp16 d | u16 scales_h | scales_l[4] | qs[128] nibbles (low = weights 0-15, high = 16-31 of
// each 32).  w = d * (ls - 32) * levels[nibble] (src/quant/quant_ref.cpp:284-300; cpu_kernels.cpp:351-384).
// The 16-entry level table lives in four registers; PRMT uses four nibbles of the data word directly as its
// selector: the low 3 bits pick among the 8 entries of a half, and with the top bit set PRMT returns the picked byte's
// sign (zero for these tables), which separates the halves (see half).
// ------------------------------------------------------------------------------------------------
template <> struct Unit<T_IQ4_XS> : UnitRun<T_IQ4_XS> {
    static constexpr int BLOCK_BYTES = 136;
    static constexpr int CODEBOOK_ENTRIES = 0;

    // levels -127,-104,-83,-65,-49,-35,-22,-10 | 1,13,25,38,53,69,89,113 as two tables of non-negative bytes: the negative
    // ones negated (127, 104, 83, 65 | 49, 35, 22, 10) and the positive ones in reverse order (113, 89, 69, 53 |
    // 38, 25, 13, 1), looked up with the data word and with its complement: see Gran<T_IQ4_XS>
    static constexpr uint32_t NL0 = 0x4153687Fu, NL1 = 0x0A162331u, HR0 = 0x35455971u, HR1 = 0x010D1926u;

    struct Row { uint32_t sc[2], hdr; };   // sc: ls - 32 of the even / odd sub-blocks, a signed byte each; hdr: fp16 d | scales_h

    static Q38B_HD void row(SP p, int, Row& r) {
        uint32_t sl;
        sp_ld64(p, 0, r.hdr, sl);
        uint32_t x = prmt(r.hdr, 0u, 0x4342u);                    // scales_h, its low byte in byte 0, its high byte in byte 2
        x = (x | (x << 4)) & 0x0F0F0F0Fu;                         // nibble k in byte k: two bits each of sub-blocks 2k, 2k + 1
        const uint32_t e = (sl & 0x0F0F0F0Fu) | ((x << 4) & 0x30303030u), o = ((sl >> 4) & 0x0F0F0F0Fu) | ((x << 2) & 0x30303030u);
        r.sc[0] = (e + 0x60606060u) ^ 0x80808080u;                // less 32: + 96 and the top bit flipped, no carries (values <= 63)
        r.sc[1] = (o + 0x60606060u) ^ 0x80808080u;
    }
    static Q38B_HD void dd(SP, const Row& r, float& d, float& m) { d = fp16_bits_to_float(r.hdr & 0xFFFFu); m = 0.0f; }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA4 = pA + 4 * e.t, pB4 = pB + 4 * e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            // The levels as two fragments of non-negative bytes, positive part and negated negative part (the two-table
            // PRMT look-up of the one-column decoder): two mma on the same activations and a subtraction cost less than
            // the masks and the merging PRMT of a single signed fragment; the tensor pipe is idle anyway.
            uint32_t b0, b1;
            const uint32_t wA = sp_ld32(pA4, 8 + 16 * s), wB = sp_ld32(pB4, 8 + 16 * s);
            sp_ld64(e.q, 32 * s, b0, b1);
            int c[4], cn[4], v[4];
            mma_k32_z(c, prmt(HR0, HR1, ~wA), prmt(HR0, HR1, ~wB), prmt(HR0, HR1, ~wA >> 16), prmt(HR0, HR1, ~wB >> 16), b0, b1);
            mma_k32_z(cn, prmt(NL0, NL1, wA), prmt(NL0, NL1, wB), prmt(NL0, NL1, wA >> 16), prmt(NL0, NL1, wB >> 16), b0, b1);
            const int scA = byte_s(A.sc[s & 1], s >> 1), scB = byte_s(B.sc[s & 1], s >> 1);
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = (i < 2 ? scA : scB) * (c[i] - cn[i]);
            emit(s, v);
        }
    }
};

// ------------------------------------------------------------------------------------------------
// Q4_K (144 bytes: fp16 d, dmin | scales[12] | qs[128]) and Q5_K (176 bytes: ... | qh[32] | qs[128]).
// w = d * sc * q - dmin * m (src/quant/quant_ref.cpp:57-76; src/cpu/cpu_kernels.cpp:386-433; Q5_K has no
// reference code: q gets a fifth bit from qh).  The min term sum_s m_s * (sum of the sub-block's activations): mins()
// from the sums that are staged beside Q8_K columns; with per-32 columns a second mma whose A operand is m_s in every slot.
// ------------------------------------------------------------------------------------------------
template <int FMT> struct UnitQ45K : UnitRun<FMT> {
    static constexpr int NBITS = FMT == T_Q5_K ? 5 : 4;
    static constexpr int BLOCK_BYTES = NBITS == 5 ? 176 : 144;
    static constexpr int CODEBOOK_ENTRIES = 0;
    static constexpr int QS_OFF = NBITS == 5 ? 48 : 16;
    static constexpr bool HAS_MIN = true;

    struct Row { uint32_t dd, sc[2], mn[2], qh[NBITS == 5 ? 2 : 1]; };

    // the minima of super-block rows A and B as k16 fragments: slots 0..7 (first digit) or 8..15 (second) hold m of the sub-blocks
    static Q38B_HD void mins(const Row& A, const Row& B, const FragEnv& e, int (&cm)[4]) {
        const uint32_t b = sp_ld32(e.bsum), lo = e.t < 2 ? 0xFFFFFFFFu : 0u;
        const uint32_t mA = (e.t & 1) ? A.mn[1] : A.mn[0], mB = (e.t & 1) ? B.mn[1] : B.mn[0];
        int hi[4];
        mma_k16_z(cm, mA & lo, mB & lo, b);
        mma_k16_z(hi, mA & ~lo, mB & ~lo, b);
#pragma unroll
        for (int i = 0; i < 4; i++) cm[i] += 64 * hi[i];
    }

    static Q38B_HD void row(SP p, int t, Row& r) {
        uint32_t hd[4];
        sp_ld128(p, 0, hd);
        r.dd = hd[0];
        const uint32_t u0 = hd[1], u1 = hd[2], u2 = hd[3];
        // 6-bit scales and mins of sub-blocks 0..3 and 4..7 as four bytes each (get_scale_min_k4, quant_ref.cpp:24-32)
        r.sc[0] = u0 & 0x3F3F3F3Fu;
        r.mn[0] = u1 & 0x3F3F3F3Fu;
        r.sc[1] = (u2 & 0x0F0F0F0Fu) | ((u0 >> 2) & 0x30303030u);
        r.mn[1] = ((u2 >> 4) & 0x0F0F0F0Fu) | ((u1 >> 2) & 0x30303030u);
        if constexpr (NBITS == 5) sp_ld64(p + 8 * t, 16, r.qh[0], r.qh[1]);
    }
    static Q38B_HD void dd(SP, const Row& r, float& d, float& m) { d = fp16_bits_to_float(r.dd & 0xFFFFu); m = fp16_bits_to_float(r.dd >> 16); }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&cm)[4], E emit) {
        const SP pA8 = pA + 8 * e.t, pB8 = pB + 8 * e.t;
#pragma unroll
        for (int pp = 0; pp < 2; pp++) {
            const int pair = 2 * h + pp;
            uint32_t wA0, wA1, wB0, wB1;
            sp_ld64(pA8, QS_OFF + 32 * pair, wA0, wA1);
            sp_ld64(pB8, QS_OFF + 32 * pair, wB0, wB1);
#pragma unroll
            for (int hn = 0; hn < 2; hn++) {   // low nibbles = sub-block 2*pair, high nibbles = 2*pair + 1
                const int s = 2 * pair + hn, j = 2 * pp + hn;
                uint32_t a0 = (wA0 >> (4 * hn)) & 0x0F0F0F0Fu, a2 = (wA1 >> (4 * hn)) & 0x0F0F0F0Fu;
                uint32_t a1 = (wB0 >> (4 * hn)) & 0x0F0F0F0Fu, a3 = (wB1 >> (4 * hn)) & 0x0F0F0F0Fu;
                if constexpr (NBITS == 5) {   // bit s of qh[l] -> bit 4 of weight l
                    a0 |= (s < 4 ? A.qh[0] << (4 - s) : A.qh[0] >> (s - 4)) & 0x10101010u;
                    a2 |= (s < 4 ? A.qh[1] << (4 - s) : A.qh[1] >> (s - 4)) & 0x10101010u;
                    a1 |= (s < 4 ? B.qh[0] << (4 - s) : B.qh[0] >> (s - 4)) & 0x10101010u;
                    a3 |= (s < 4 ? B.qh[1] << (4 - s) : B.qh[1] >> (s - 4)) & 0x10101010u;
                }
                uint32_t b0, b1;
                sp_ld64(e.q, 32 * s, b0, b1);
                int c[4], v[4];
                mma_k32_z(c, a0, a1, a2, a3, b0, b1);
                const int scA = byte_u(A.sc[h], j), scB = byte_u(B.sc[h], j);
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = (i < 2 ? scA : scB) * c[i];
                if constexpr (!TABLES) {   // (with staged sums: mins)
                    const uint32_t mA = prmt(A.mn[h], 0u, 0x1111u * (uint32_t)j), mB = prmt(B.mn[h], 0u, 0x1111u * (uint32_t)j);
                    mma_k32(cm, mA, mB, mA, mB, b0, b1);
                }
                emit(s, v);
            }
        }
    }
};
template <> struct Unit<T_Q4_K> : UnitQ45K<T_Q4_K> {};
template <> struct Unit<T_Q5_K> : UnitQ45K<T_Q5_K> {};

// ------------------------------------------------------------------------------------------------
// Q6_K: 210 bytes = ql[128] | qh[64] | int8 scales[16] | fp16 d.  w = d * sc[group of 16] * (q - 32)
// (src/quant/quant_ref.cpp:78-103; src/cpu/cpu_kernels.cpp:479-515).  One k16 mma per 16-weight group.
// Half h of the block = weights 128h..128h+127; lane t reads ql bytes l..l+3 and l+32..l+35 and qh bytes l..l+3
// for l = 16e + 4t (e = 0, 1), which hold four groups (j = 0..3): weights 128h + 32j + 16e + 4t .. +3.
// ------------------------------------------------------------------------------------------------
template <> struct Unit<T_Q6_K> : UnitRun<T_Q6_K> {
    static constexpr int BLOCK_BYTES = 210;
    static constexpr int CODEBOOK_ENTRIES = 0;
    static constexpr int ACT_STEP = 4;
    struct Row {};
    static Q38B_HD void row(SP, int, Row&) {}
    static Q38B_HD void dd(SP p, const Row&, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(p, 208)); m = 0.0f; }

    // four 6-bit weights per byte lane, minus 32, as int8
    static Q38B_HD uint32_t q6(uint32_t low4, uint32_t high2_at_bit4) {
        const uint32_t v = (low4 & 0x0F0F0F0Fu) | (high2_at_bit4 & 0x30303030u);
        return (v + 0x60606060u) ^ 0x80808080u;   // +96 then flip the top bit = -32 per byte, no carries (v <= 63)
    }

    static Q38B_HD void row_words(SP p4t, int h, int e, uint32_t (&w)[4]) {
        const uint32_t qa = ld_u32_a2(p4t, 64 * h + 16 * e), qb = ld_u32_a2(p4t, 64 * h + 32 + 16 * e);
        const uint32_t qh = ld_u32_a2(p4t, 128 + 32 * h + 16 * e);
        w[0] = q6(qa, qh << 4);
        w[1] = q6(qb, qh << 2);
        w[2] = q6(qa >> 4, qh);
        w[3] = q6(qb >> 4, qh >> 2);
    }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row&, const Row&, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA4 = pA + 4 * e.t, pB4 = pB + 4 * e.t;
        uint32_t wA[2][4], wB[2][4];
#pragma unroll
        for (int g = 0; g < 2; g++) { row_words(pA4, h, g, wA[g]); row_words(pB4, h, g, wB[g]); }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int v[4] = {0, 0, 0, 0};
#pragma unroll
            for (int g = 0; g < 2; g++) {
                int c[4];
                mma_k16_z(c, wA[g][j], wB[g][j], sp_ld32(e.q, 128 * h + 32 * j + 16 * g));
                const int scA = sp_ld8s(pA, 192 + 8 * h + 2 * j + g), scB = sp_ld8s(pB, 192 + 8 * h + 2 * j + g);
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] += (i < 2 ? scA : scB) * c[i];
            }
            emit(4 * h + j, v);
        }
    }
};

// ------------------------------------------------------------------------------------------------
// Q8_0: eight 34-byte blocks (fp16 d | int8 qs[32]) per 256 weights; w = d * q (src/quant/quant_ref.cpp:302-308;
// the reference has no dot kernel for it).  The float scale changes every 32 weights (SCALE32), so each mma result is
// converted and accumulated in float.
// ------------------------------------------------------------------------------------------------
template <> struct Unit<T_Q8_0> : UnitRun<T_Q8_0> {
    static constexpr int BLOCK_BYTES = 272;   // bytes per 256 weights
    static constexpr int CODEBOOK_ENTRIES = 0;
    static constexpr bool SCALE32 = true;
    struct Row {};
    static Q38B_HD void row(SP, int, Row&) {}
    static Q38B_HD void dd(SP, const Row&, float& d, float& m) { d = 0.0f; m = 0.0f; }
    static Q38B_HD float d32(SP p, int s) { return fp16_bits_to_float(sp_ld16(p, 34 * s)); }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row&, const Row&, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA8 = pA + 8 * e.t, pB8 = pB + 8 * e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            uint32_t b0, b1;
            sp_ld64(e.q, 32 * s, b0, b1);
            int c[4];
            mma_k32_z(c, ld_u32_a2(pA8, 34 * s + 2), ld_u32_a2(pB8, 34 * s + 2), ld_u32_a2(pA8, 34 * s + 6), ld_u32_a2(pB8, 34 * s + 6), b0, b1);
            emit(s, c);
        }
    }
};

// ------------------------------------------------------------------------------------------------
// The reference's other six formats (block layouts: src/quant/quant_formats.h:92,97-99,102-103; integer sums of
// src/cpu/cpu_kernels.cpp:191-349, 435-477).  Their grids hold eight values out of three levels per entry: shared memory keeps
// an entry as eight bytes in several copies (magnitudes 8, 25, 43; for IQ1 eight times the level -1, 0, 1), codebooks.inc as
// eight 2-bit level indices (CODE16_ENTRIES).
// ------------------------------------------------------------------------------------------------
// The scale of IQ2_XS, IQ2_S and IQ1_M changes every 16 weights, a grid entry holds eight: lanes 0, 1 of a row hold the first
// half of a sub-block and lanes 2, 3 the second.  Two mma with the same weights, each with the other half's activations zero.
Q38B_HD void mma_halves(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, const FragEnv& e, int off, int (&c0)[4], int (&c1)[4]) {
    uint32_t b0, b1, b2, b3;
    sp_ld64(e.q_half[0], off, b0, b1);
    sp_ld64(e.q_half[1], off, b2, b3);
    mma_k32_z(c0, a0, a1, a2, a3, b0, b1);
    mma_k32_z(c1, a0, a1, a2, a3, b2, b3);
}
// eight-byte grid entry number idx
Q38B_HD void grid8(const FragEnv& e, uint32_t idx, uint32_t& lo, uint32_t& hi) { sp_ld64(e.cb + (int)(idx << e.cb_shift), 0, lo, hi); }

// IQ2_XXS: 66 bytes = fp16 d | 8 x (4 grid indices, u32 of 4 x 7 sign bits + 4-bit scale)
template <> struct Unit<T_IQ2_XXS> : UnitRun<T_IQ2_XXS> {
    static constexpr int BLOCK_BYTES = 66, CODEBOOK_ENTRIES = 0, CODE16_ENTRIES = 256;
    static constexpr float FACTOR = 0.125f;
    struct Row { uint32_t aux[2]; };
    static Q38B_HD void row(SP p, int t, Row& r) {
        r.aux[0] = ld_u32_a2(p + 8 * t, 6);
        r.aux[1] = ld_u32_a2(p + 8 * t, 38);
    }
    static Q38B_HD void dd(SP p, const Row&, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(p, 0)); m = 0.0f; }
    template <bool TABLES>
    static Q38B_HD void weights(SP pt, int s, uint32_t aux, const FragEnv& e, Signed8& w, int& scale) {
        grid8(e, sp_ld8(pt, 2 + 8 * s), w.g0, w.g1);
        sign_masks7_at<TABLES>(e, aux, 7 * e.t, w.m0, w.m1);
        scale = (int)(2u * (aux >> 28) + 1u);
    }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA1 = pA + e.t, pB1 = pB + e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            Signed8 wA, wB;
            int scA, scB, v[4];
            weights<TABLES>(pA1, s, quad_shfl(A.aux[h], j), e, wA, scA);
            weights<false>(pB1, s, quad_shfl(B.aux[h], j), e, wB, scB);
            uint32_t b0, b1;
            sp_ld64(e.q, 32 * s, b0, b1);
            mma_signed(wA, wB, b0, b1, scA, scB, v);
            emit(s, v);
        }
    }
};

// IQ2_XS: 74 bytes = fp16 d | 32 x u16 (9-bit grid index, 7 sign bits) | scales[8] (a nibble per 16 weights)
template <> struct Unit<T_IQ2_XS> : UnitRun<T_IQ2_XS> {
    static constexpr int BLOCK_BYTES = 74, CODEBOOK_ENTRIES = 0, CODE16_ENTRIES = 512;
    static constexpr float FACTOR = 0.125f;
    struct Row { uint32_t sc[2]; };
    static Q38B_HD void row(SP p, int, Row& r) { r.sc[0] = ld_u32_a2(p, 66); r.sc[1] = ld_u32_a2(p, 70); }
    static Q38B_HD void dd(SP p, const Row&, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(p, 0)); m = 0.0f; }
    template <bool TABLES>
    static Q38B_HD void weights(SP p2t, int s, const FragEnv& e, uint32_t& w0, uint32_t& w1) {
        const uint32_t qv = sp_ld16(p2t, 2 + 8 * s);
        uint32_t g0, g1, m0, m1;
        grid8(e, qv & 511u, g0, g1);
        if constexpr (TABLES) sp_ld64(e.sgn + (int)((qv >> (9 - SIGN_STRIDE_LOG2)) & (127u << SIGN_STRIDE_LOG2)), 0, m0, m1);
        else sign_masks7(qv >> 9, m0, m1);
        w0 = negate_bytes(g0, m0);
        w1 = negate_bytes(g1, m1);
    }
    // the scale 2 n + 1 of nibble k of the sub-blocks' scale bytes w
    static Q38B_HD int scale(uint32_t w, int k) { return (int)(((k == 0 ? (w << 1) : (w >> (4 * k - 1))) & 0x1Eu) + 1u); }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA2 = pA + 2 * e.t, pB2 = pB + 2 * e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            uint32_t a0, a1, a2, a3;
            weights<TABLES>(pA2, s, e, a0, a2);
            weights<false>(pB2, s, e, a1, a3);   // (one row by look-up, one computed: see sign_masks7_at)
            int c0[4], c1[4], v[4];
            mma_halves(a0, a1, a2, a3, e, 32 * s, c0, c1);
            const int sA0 = scale(A.sc[h], 2 * j), sA1 = scale(A.sc[h], 2 * j + 1), sB0 = scale(B.sc[h], 2 * j), sB1 = scale(B.sc[h], 2 * j + 1);
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = (i < 2 ? sA0 : sB0) * c0[i] + (i < 2 ? sA1 : sB1) * c1[i];
            emit(s, v);
        }
    }
};

// IQ2_S: 82 bytes = fp16 d | qs[32] | signs[32] | qh[8] (two high index bits a group) | scales[8]
template <> struct Unit<T_IQ2_S> : UnitRun<T_IQ2_S> {
    static constexpr int BLOCK_BYTES = 82, CODEBOOK_ENTRIES = 0, CODE16_ENTRIES = 1024;
    static constexpr float FACTOR = 0.125f;
    struct Row { uint32_t sc[2], qh[2]; };   // qh: shifted so that this lane's two bits of sub-block j are bits 8 j, 8 j + 1
    static Q38B_HD void row(SP p, int t, Row& r) {
        r.qh[0] = ld_u32_a2(p, 66) >> (2 * t);
        r.qh[1] = ld_u32_a2(p, 70) >> (2 * t);
        r.sc[0] = ld_u32_a2(p, 74);
        r.sc[1] = ld_u32_a2(p, 78);
    }
    static Q38B_HD void dd(SP p, const Row&, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(p, 0)); m = 0.0f; }
    static Q38B_HD void weights(SP pt, int s, uint32_t qh, const FragEnv& e, uint32_t& w0, uint32_t& w1) {
        const int j = s & 3;
        uint32_t g0, g1, m0, m1;
        grid8(e, sp_ld8(pt, 2 + 4 * s) | ((j == 0 ? (qh << 8) : (qh >> (8 * j - 8))) & 0x300u), g0, g1);
        sign_masks8(sp_ld8(pt, 34 + 4 * s), m0, m1);
        w0 = negate_bytes(g0, m0);
        w1 = negate_bytes(g1, m1);
    }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA1 = pA + e.t, pB1 = pB + e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            uint32_t a0, a1, a2, a3;
            weights(pA1, s, A.qh[h], e, a0, a2);
            weights(pB1, s, B.qh[h], e, a1, a3);
            int c0[4], c1[4], v[4];
            mma_halves(a0, a1, a2, a3, e, 32 * s, c0, c1);
            using X = Unit<T_IQ2_XS>;
            const int sA0 = X::scale(A.sc[h], 2 * j), sA1 = X::scale(A.sc[h], 2 * j + 1), sB0 = X::scale(B.sc[h], 2 * j), sB1 = X::scale(B.sc[h], 2 * j + 1);
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = (i < 2 ? sA0 : sB0) * c0[i] + (i < 2 ? sA1 : sB1) * c1[i];
            emit(s, v);
        }
    }
};

// IQ1_S: 50 bytes = fp16 d | qs[32] | qh[8] u16 (4 x 3 high index bits, 3-bit scale, sign of the delta).  A weight is
// 8 (level - 1) + 1 or - 1: the delta is a second mma whose A operand is 1 or -1 in every slot.
template <> struct Unit<T_IQ1_S> : UnitRun<T_IQ1_S> {
    static constexpr int BLOCK_BYTES = 50, CODEBOOK_ENTRIES = 0, CODE16_ENTRIES = 2048;
    static constexpr float FACTOR = 0.125f;
    struct Row {};
    static Q38B_HD void row(SP, int, Row&) {}
    static Q38B_HD void dd(SP p, const Row&, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(p, 0)); m = 0.0f; }
    static Q38B_HD void weights(SP p, SP pt, int s, const FragEnv& e, uint32_t& g0, uint32_t& g1, uint32_t& delta, int& scale) {
        const uint32_t qh = sp_ld16(p, 34 + 2 * s);
        grid8(e, sp_ld8(pt, 2 + 4 * s) | (((qh >> (3 * e.t)) & 7u) << 8), g0, g1);
        delta = (qh & 0x8000u) ? 0xFFFFFFFFu : 0x01010101u;
        scale = (int)(((qh >> 11) & 0xEu) + 1u);
    }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row&, const Row&, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA1 = pA + e.t, pB1 = pB + e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            uint32_t a0, a1, a2, a3, dA, dB, b0, b1;
            int scA, scB, c[4], v[4];
            weights(pA, pA1, s, e, a0, a2, dA, scA);
            weights(pB, pB1, s, e, a1, a3, dB, scB);
            sp_ld64(e.q, 32 * s, b0, b1);
            mma_k32_z(c, a0, a1, a2, a3, b0, b1);
            mma_k32(c, dA, dB, dA, dB, b0, b1);
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = (i < 2 ? scA : scB) * c[i];
            emit(s, v);
        }
    }
};

// IQ1_M: 56 bytes = qs[32] | qh[16] (per group of eight: 3 high index bits, sign of the delta) | scales[8]: four u16 with 3-bit
// scales per 16 weights and, in their top nibbles, the fp16 super-scale
template <> struct Unit<T_IQ1_M> : UnitRun<T_IQ1_M> {
    static constexpr int BLOCK_BYTES = 56, CODEBOOK_ENTRIES = 0, CODE16_ENTRIES = 2048;
    static constexpr float FACTOR = 0.125f;
    struct Row { uint32_t sw[4]; };
    static Q38B_HD void row(SP p, int, Row& r) {
#pragma unroll
        for (int i = 0; i < 4; i++) r.sw[i] = sp_ld16(p, 48 + 2 * i);
    }
    static Q38B_HD void dd(SP, const Row& r, float& d, float& m) {
        d = fp16_bits_to_float((r.sw[0] >> 12) | ((r.sw[1] >> 8) & 0x00F0u) | ((r.sw[2] >> 4) & 0x0F00u) | (r.sw[3] & 0xF000u));
        m = 0.0f;
    }
    static Q38B_HD void weights(SP p, SP pt, int s, const FragEnv& e, uint32_t& g0, uint32_t& g1, uint32_t& delta) {
        const uint32_t hn = sp_ld16(p, 32 + 2 * s) >> (4 * e.t);
        grid8(e, sp_ld8(pt, 4 * s) | ((hn & 7u) << 8), g0, g1);
        delta = (hn & 8u) ? 0xFFFFFFFFu : 0x01010101u;
    }
    static Q38B_HD int scale(const Row& r, int s, int h) {   // half h of sub-block s
        const int at = 6 * (s & 1) + 3 * h;
        return (int)(((at == 0 ? (r.sw[s >> 1] << 1) : (r.sw[s >> 1] >> (at - 1))) & 0xEu) + 1u);
    }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&)[4], E emit) {
        const SP pA1 = pA + e.t, pB1 = pB + e.t;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            uint32_t a0, a1, a2, a3, dA, dB, b0, b1, b2, b3;
            weights(pA, pA1, s, e, a0, a2, dA);
            weights(pB, pB1, s, e, a1, a3, dB);
            sp_ld64(e.q_half[0], 32 * s, b0, b1);
            sp_ld64(e.q_half[1], 32 * s, b2, b3);
            int c0[4], c1[4], v[4];
            mma_k32_z(c0, a0, a1, a2, a3, b0, b1);
            mma_k32(c0, dA, dB, dA, dB, b0, b1);
            mma_k32_z(c1, a0, a1, a2, a3, b2, b3);
            mma_k32(c1, dA, dB, dA, dB, b2, b3);
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = scale(i < 2 ? A : B, s, 0) * c0[i] + scale(i < 2 ? A : B, s, 1) * c1[i];
            emit(s, v);
        }
    }
};

// Q2_K: 84 bytes = scales[16] (low nibble scale, high nibble min, per 16 weights) | qs[64] | fp16 d | fp16 dmin; sub-block
// 4n + j = bits 2j, 2j + 1 of the 32 bytes qs[32n ..]; w = d * sc * q - dmin * m.  Rows must be 4-byte aligned.
template <> struct Unit<T_Q2_K> : UnitRun<T_Q2_K> {
    static constexpr int BLOCK_BYTES = 84, CODEBOOK_ENTRIES = 0, CODE16_ENTRIES = 0;
    static constexpr bool HAS_MIN = true;
    static constexpr int ACT_STEP = 4;
    struct Row { uint32_t sc[4], dd; };
    static Q38B_HD void mins(const Row& A, const Row& B, const FragEnv& e, int (&cm)[4]) {
        const uint32_t wA = e.t == 0 ? A.sc[0] : e.t == 1 ? A.sc[1] : e.t == 2 ? A.sc[2] : A.sc[3];
        const uint32_t wB = e.t == 0 ? B.sc[0] : e.t == 1 ? B.sc[1] : e.t == 2 ? B.sc[2] : B.sc[3];
        const uint32_t mA = (wA >> 4) & 0x0F0F0F0Fu, mB = (wB >> 4) & 0x0F0F0F0Fu;
        int hi[4];
        mma_k16_z(cm, mA, mB, sp_ld32(e.bsum));
        mma_k16_z(hi, mA, mB, sp_ld32(e.bsum, 16));
#pragma unroll
        for (int i = 0; i < 4; i++) cm[i] += 64 * hi[i];
    }
    static Q38B_HD void row(SP p, int, Row& r) {
#pragma unroll
        for (int i = 0; i < 4; i++) r.sc[i] = sp_ld32(p, 4 * i);
        r.dd = sp_ld32(p, 80);
    }
    static Q38B_HD void dd(SP, const Row& r, float& d, float& m) { d = fp16_bits_to_float(r.dd & 0xFFFFu); m = fp16_bits_to_float(r.dd >> 16); }
    template <bool TABLES, class E>
    static Q38B_HD void half(const Row& A, const Row& B, SP pA, SP pB, int h, const FragEnv& e, int (&cm)[4], E emit) {
        const SP pA4 = pA + 4 * e.t, pB4 = pB + 4 * e.t;
        uint32_t wA[2], wB[2];
#pragma unroll
        for (int g = 0; g < 2; g++) { wA[g] = sp_ld32(pA4, 16 + 32 * h + 16 * g); wB[g] = sp_ld32(pB4, 16 + 32 * h + 16 * g); }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int s = 4 * h + j;
            int v[4] = {0, 0, 0, 0};
#pragma unroll
            for (int g = 0; g < 2; g++) {
                const int k = 2 * (s & 1) + g;                      // scale byte of the group in its word
                const uint32_t b0 = sp_ld32(e.q, 32 * s + 16 * g);
                const uint32_t nA = A.sc[s >> 1] >> (8 * k), nB = B.sc[s >> 1] >> (8 * k);
                int c[4];
                mma_k16_z(c, (wA[g] >> (2 * j)) & 0x03030303u, (wB[g] >> (2 * j)) & 0x03030303u, b0);
                if constexpr (!TABLES) mma_k16(cm, ((nA >> 4) & 0xFu) * 0x01010101u, ((nB >> 4) & 0xFu) * 0x01010101u, b0);
                const int scA = (int)(nA & 0xFu), scB = (int)(nB & 0xFu);
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] += (i < 2 ? scA : scB) * c[i];
            }
            emit(s, v);
        }
    }
};

// 16-bit grid codes a format keeps in shared memory (0 for the formats without such a table)
Q38B_HD constexpr int code16_entries(int fmt) {
    return fmt == T_IQ2_XXS ? 256 : fmt == T_IQ2_XS ? 512 : fmt == T_IQ2_S ? 1024 : (fmt == T_IQ1_S || fmt == T_IQ1_M) ? 2048 : 0;
}
// formats whose several columns give the one-column kernel's bits (they are never cut into K-parts)
Q38B_HD constexpr bool one_column_only(int fmt) {
    return fmt == T_Q2_K || fmt == T_IQ2_XXS || fmt == T_IQ2_XS || fmt == T_IQ2_S || fmt == T_IQ1_S || fmt == T_IQ1_M;
}

// bytes of one 256-weight super-block
Q38B_HD constexpr int block_bytes(int fmt) {
    switch (fmt) {
        case T_Q8_0: return 272; case T_Q4_K: return 144; case T_Q5_K: return 176; case T_Q6_K: return 210;
        case T_IQ3_XXS: return 98; case T_IQ3_S: return 110; case T_IQ4_XS: return 136;
        case T_Q2_K: return 84; case T_IQ2_XXS: return 66; case T_IQ2_XS: return 74; case T_IQ2_S: return 82;
        case T_IQ1_S: return 50; case T_IQ1_M: return 56; default: return 0;
    }
}

}  // namespace q38b
