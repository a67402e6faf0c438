// q38b_expand.cuh -- 32 weights of a GGUF block, staged in shared memory in their file layout, as fp32, fp16 or bf16.
//
// Every format is brought to the same form first: 32 unsigned bytes u (eight words), for the sign-magnitude formats 32
// sign bits, and per half (16 weights) a scale and an offset.  A byte becomes a float with one PRMT (under the exponent
// of 2^15, where one unit of byte 1 is 1.0) and an exact subtraction; the multiplication and, for the K-quants, the
// subtraction of the minimum are the float operations of dequantize_row_ref (src/quant/quant_ref.cpp:57-103, 165-308 of
// the reference project), each rounded as there (d * sc and d1 * q are exact in fp32, so the K-quants' multiply and
// subtract are one fused operation with the same result).  Two results are rounded and packed by one instruction and the
// signs are XOR-ed into the packed pair: a multiplication moves two sign bits to bits 15 and 31.
//
// A thread works on whole words where the byte-wise dequantizer it replaces issued a load and a shift per weight; blocks
// of most formats are only 2-byte aligned, so words are read aligned and funnel-shifted.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdint>

#include "q38b_decode1.cuh"

namespace q38b {

// grid entries a format's expander looks up in shared memory, 4-byte words per entry, and copies of the table: lanes of a
// warp meet on a bank less often with several copies (entry e, copy r at word (e * copies + r) * words); 8 KB where more
// than one copy fits
struct GridTable { int entries, words, copies; };
__host__ __device__ constexpr GridTable grid_table(int fmt) {
    return fmt == T_IQ3_XXS ? GridTable{256, 1, 8} : fmt == T_IQ3_S ? GridTable{512, 1, 4} : fmt == T_IQ2_XXS ? GridTable{256, 2, 4}
         : fmt == T_IQ2_XS ? GridTable{512, 2, 2} : fmt == T_IQ2_S ? GridTable{1024, 2, 1}
         : fmt == T_IQ1_S || fmt == T_IQ1_M ? GridTable{2048, 2, 1} : GridTable{0, 0, 0};
}
__host__ __device__ constexpr int grid_table_bytes(int fmt) { return grid_table(fmt).entries * grid_table(fmt).words * grid_table(fmt).copies * 4; }

// Fills the table with threads t = 0 .. n - 1; `src`: the context's device table of the format (32-bit grid words, or two
// 16-bit codes of eight 2-bit level numbers per word).
template <int FMT>
__device__ __forceinline__ void fill_grid_table(uint32_t* tab, const uint32_t* src, int t, int n) {
    constexpr GridTable G = grid_table(FMT);
#pragma unroll 8
    for (int e = t; e < G.entries; e += n) {   // (a thread's loads go out together: one after the other they were most of a small call)
        if (G.words == 1) {
            const uint32_t w = src[e];
            for (int r = 0; r < G.copies; r++) tab[e * G.copies + r] = w;
        } else {
            const uint32_t code = (src[e >> 1] >> (16 * (e & 1))) & 0xFFFFu;
            constexpr uint32_t LEVELS = (FMT == T_IQ1_S || FMT == T_IQ1_M) ? 0x00020100u : 0x002B1908u;   // 0, 1, 2 (minus one: the weight) or 8, 25, 43
            const uint32_t lo = prmt(LEVELS, 0u, sel_from_codes(code & 0xFFu)), hi = prmt(LEVELS, 0u, sel_from_codes(code >> 8));
            for (int r = 0; r < G.copies; r++) {
                tab[(e * G.copies + r) * 2] = lo;
                tab[(e * G.copies + r) * 2 + 1] = hi;
            }
        }
    }
}

// N words from a 2-byte aligned address (aligned loads and funnel shifts; up to four bytes past the last word are read)
template <int N>
__device__ __forceinline__ void words_a2(const uint8_t* p, uint32_t (&w)[N]) {
    const uint32_t mis = (uint32_t)(uintptr_t)p & 2u;
    const uint32_t* q = (const uint32_t*)(p - mis);
    uint32_t prev = q[0];
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint32_t next = q[i + 1];
        w[i] = __funnelshift_r(prev, next, 8u * mis);
        prev = next;
    }
}
// N words from an address that is a multiple of ALIGN = 16, 4 or 2
template <int N, int ALIGN>
__device__ __forceinline__ void words_of(const uint8_t* p, uint32_t (&w)[N]) {
    if constexpr (ALIGN == 16) {
        static_assert(N % 4 == 0, "whole 16-byte loads");
#pragma unroll
        for (int i = 0; i < N / 4; i++) {
            const uint4 v = *(const uint4*)(p + 16 * i);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    } else if constexpr (ALIGN == 4) {
#pragma unroll
        for (int i = 0; i < N; i++) w[i] = *(const uint32_t*)(p + 4 * i);
    } else {
        words_a2<N>(p, w);
    }
}
__device__ __forceinline__ float s_f16(const uint8_t* p) { return __half2float(__ushort_as_half(*(const unsigned short*)p)); }
__device__ __forceinline__ uint32_t s_u16(const uint8_t* p) { return *(const uint16_t*)p; }

// sub-block in common form: value k = (u_k + off) * a, negated where its sign bit is set; AFFINE: u_k * a - c
struct Sub32 {
    uint32_t u[8];
    uint32_t sign;
    float a[2], c[2];     // per half
    float off[4];         // per eight weights
};
enum : int { FORM_MAGNITUDE = 0, FORM_AFFINE = 1, FORM_OFFSET = 2 };
__host__ __device__ constexpr int expand_form(int fmt) {
    return fmt == T_Q4_K || fmt == T_Q5_K || fmt == T_Q2_K ? FORM_AFFINE : fmt == T_Q6_K || fmt == T_Q8_0 || fmt == T_IQ1_S || fmt == T_IQ1_M ? FORM_OFFSET : FORM_MAGNITUDE;
}
// the ALIGNED variants exist for the formats whose blocks keep an alignment of more than 2 bytes (16, 16, 8, 4)
__host__ __device__ constexpr int expand_alignment(int fmt) { return fmt == T_Q4_K || fmt == T_Q5_K ? 16 : fmt == T_IQ4_XS ? 8 : fmt == T_Q2_K ? 4 : 2; }

// s7: seven sign bits of eight weights; the eighth makes their number even
__device__ __forceinline__ uint32_t sign8(uint32_t s7) { return s7 | ((uint32_t)__popc(s7) << 7); }   // (bits above 7 are garbage)

// sub-block s (0..7) of the 256-weight block at `b` (shared memory); `tab`: the grid table, already moved to this lane's copy
template <int FMT, bool ALIGNED>
__device__ __forceinline__ void load_sub32(const uint8_t* b, int s, const uint32_t* tab, Sub32& o) {
    constexpr GridTable G = grid_table(FMT);
    constexpr int AL = ALIGNED ? expand_alignment(FMT) : 2;   // what `b` is a multiple of
    o.sign = 0u;
    if constexpr (FMT == T_Q8_0) {
        const uint8_t* p = b + 34 * s;
        words_a2<8>(p + 2, o.u);
#pragma unroll
        for (int i = 0; i < 8; i++) o.u[i] ^= 0x80808080u;
        o.a[0] = o.a[1] = s_f16(p);
#pragma unroll
        for (int i = 0; i < 4; i++) o.off[i] = -128.0f;
    } else if constexpr (FMT == T_Q4_K || FMT == T_Q5_K) {
        uint32_t h[4];
        words_of<4, AL>(b, h);
        const float d = __half2float(__ushort_as_half((unsigned short)h[0])), mn = __half2float(__ushort_as_half((unsigned short)(h[0] >> 16)));
        // 6-bit scales and minima (get_scale_min_k4, src/quant/quant_ref.cpp:24-32): four bytes of the half of the block
        const uint32_t sc4 = s >= 4 ? ((h[3] & 0x0F0F0F0Fu) | ((h[1] >> 2) & 0x30303030u)) : (h[1] & 0x3F3F3F3Fu);
        const uint32_t mn4 = s >= 4 ? (((h[3] >> 4) & 0x0F0F0F0Fu) | ((h[2] >> 2) & 0x30303030u)) : (h[2] & 0x3F3F3F3Fu);
        o.a[0] = o.a[1] = __fmul_rn(d, (float)((sc4 >> (8 * (s & 3))) & 0xFFu));
        o.c[0] = o.c[1] = __fmul_rn(mn, (float)((mn4 >> (8 * (s & 3))) & 0xFFu));
        words_of<8, AL>(b + (FMT == T_Q5_K ? 48 : 16) + 32 * (s >> 1), o.u);
#pragma unroll
        for (int i = 0; i < 8; i++) o.u[i] = (o.u[i] >> (4 * (s & 1))) & 0x0F0F0F0Fu;
        if constexpr (FMT == T_Q5_K) {
            uint32_t qh[8];
            words_of<8, AL>(b + 16, qh);
#pragma unroll
            for (int i = 0; i < 8; i++) o.u[i] |= ((qh[i] >> s) << 4) & 0x10101010u;
        }
    } else if constexpr (FMT == T_Q6_K) {
        const int h = s >> 2, j = s & 3;
        uint32_t ql[8], qh[8];
        words_a2<8>(b + 64 * h + 32 * (j & 1), ql);
        words_a2<8>(b + 128 + 32 * h, qh);
#pragma unroll
        for (int i = 0; i < 8; i++) o.u[i] = ((ql[i] >> (4 * (j >> 1))) & 0x0F0F0F0Fu) | (((qh[i] >> (2 * j)) << 4) & 0x30303030u);
        const float d = s_f16(b + 208);
        const int8_t* sc = (const int8_t*)(b + 192 + 8 * h + 2 * j);
        o.a[0] = __fmul_rn(d, (float)sc[0]);
        o.a[1] = __fmul_rn(d, (float)sc[1]);
#pragma unroll
        for (int i = 0; i < 4; i++) o.off[i] = -32.0f;
    } else if constexpr (FMT == T_Q2_K) {            // src/quant/quant_ref.cpp:33-55
        const int n = s >> 2, j = s & 3;
        words_of<8, AL>(b + 16 + 32 * n, o.u);
#pragma unroll
        for (int i = 0; i < 8; i++) o.u[i] = (o.u[i] >> (2 * j)) & 0x03030303u;
        const float d = s_f16(b + 80), mn = s_f16(b + 82);
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const uint32_t sc = b[2 * s + half];
            o.a[half] = __fmul_rn(d, (float)(sc & 0xFu));
            o.c[half] = __fmul_rn(mn, (float)(sc >> 4));
        }
    } else if constexpr (FMT == T_IQ4_XS) {
        // magnitudes of the 16 levels by two PRMT look-ups with the nibbles as selectors (see Unit<T_IQ4_XS>): one of the two
        // is zero.  Low nibbles are weights 0..15, high nibbles 16..31; nibbles 0..7 are the negative levels.
        using U = Unit<T_IQ4_XS>;
        uint32_t q[4];
        if (ALIGNED) {
            const uint2 v0 = *(const uint2*)(b + 8 + 16 * s), v1 = *(const uint2*)(b + 16 + 16 * s);
            q[0] = v0.x; q[1] = v0.y; q[2] = v1.x; q[3] = v1.y;
        } else {
            words_a2<4>(b + 8 + 16 * s, q);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            // selectors in nibble order (w0 low, w0 high, w1 low, ...): two words hold bytes (l0 h0 l1 h1) and (l2 h2 l3 h3)
            const uint32_t x = prmt(U::HR0, U::HR1, ~q[i]) | prmt(U::NL0, U::NL1, q[i]);
            const uint32_t y = prmt(U::HR0, U::HR1, ~q[i] >> 16) | prmt(U::NL0, U::NL1, q[i] >> 16);
            o.u[i] = prmt(x, y, 0x6420u);
            o.u[4 + i] = prmt(x, y, 0x7531u);
        }
        // sign bits: bit 3 (bit 7) of byte k of word i is clear where weight 4 i + k (16 + 4 i + k) is negative; a
        // multiplication gathers the four bits of a word
        uint32_t sg = 0u;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t lo = (~q[i] >> 3) & 0x01010101u, hi = (~q[i] >> 7) & 0x01010101u;
            sg |= ((lo * 0x10204080u) >> 28) << (4 * i);
            sg |= ((hi * 0x10204080u) >> 28) << (16 + 4 * i);
        }
        o.sign = sg;
        const uint32_t sh = s_u16(b + 2);
        const int ls = (int)(((b[4 + (s >> 1)] >> (4 * (s & 1))) & 0xFu) | (((sh >> (2 * s)) & 3u) << 4));
        o.a[0] = o.a[1] = __fmul_rn(s_f16(b), (float)(ls - 32));
    } else if constexpr (FMT == T_IQ3_XXS || FMT == T_IQ3_S) {
        uint32_t q[2];
        words_a2<2>(b + 2 + 8 * s, q);
        const float d = s_f16(b);
        if constexpr (FMT == T_IQ3_XXS) {
            uint32_t aux[1];
            words_a2<1>(b + 66 + 4 * s, aux);
            o.a[0] = o.a[1] = __fmul_rn(__fmul_rn(d, __fadd_rn(0.5f, (float)(aux[0] >> 28))), 0.5f);
#pragma unroll
            for (int l = 0; l < 4; l++) o.sign |= (sign8((aux[0] >> (7 * l)) & 127u) & 0xFFu) << (8 * l);
        } else {
            uint32_t sg[1];
            words_a2<1>(b + 74 + 4 * s, sg);
            o.sign = sg[0];
            const uint32_t ls = (b[106 + (s >> 1)] >> (4 * (s & 1))) & 0xFu;
            o.a[0] = o.a[1] = __fmul_rn(d, (float)(1 + 2 * (int)ls));
        }
        const uint32_t qh = FMT == T_IQ3_S ? b[66 + s] : 0u;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            uint32_t e = (q[i >> 2] >> (8 * (i & 3))) & 0xFFu;
            if (FMT == T_IQ3_S) e |= ((qh >> i) & 1u) << 8;
            o.u[i] = tab[e * G.copies];
        }
    } else {
        uint32_t e[4];
        if constexpr (FMT == T_IQ2_XXS) {            // src/quant/quant_ref.cpp:105-168
            uint32_t w[2];
            words_a2<2>(b + 2 + 8 * s, w);
#pragma unroll
            for (int l = 0; l < 4; l++) {
                e[l] = (w[0] >> (8 * l)) & 0xFFu;
                o.sign |= (sign8((w[1] >> (7 * l)) & 127u) & 0xFFu) << (8 * l);
            }
            o.a[0] = o.a[1] = __fmul_rn(__fmul_rn(s_f16(b), __fadd_rn(0.5f, (float)(w[1] >> 28))), 0.25f);
        } else if constexpr (FMT == T_IQ2_XS || FMT == T_IQ2_S) {
            const uint32_t sc = b[(FMT == T_IQ2_XS ? 66 : 74) + s];
            const float d = s_f16(b);
            o.a[0] = __fmul_rn(__fmul_rn(d, __fadd_rn(0.5f, (float)(sc & 0xFu))), 0.25f);
            o.a[1] = __fmul_rn(__fmul_rn(d, __fadd_rn(0.5f, (float)(sc >> 4))), 0.25f);
            if constexpr (FMT == T_IQ2_XS) {
                uint32_t w[2];
                words_a2<2>(b + 2 + 8 * s, w);
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    const uint32_t v = (w[l >> 1] >> (16 * (l & 1))) & 0xFFFFu;
                    e[l] = v & 511u;
                    o.sign |= (sign8(v >> 9) & 0xFFu) << (8 * l);
                }
            } else {
                uint32_t w[1], sg[1];
                words_a2<1>(b + 2 + 4 * s, w);
                words_a2<1>(b + 34 + 4 * s, sg);
                const uint32_t qh = b[66 + s];
#pragma unroll
                for (int l = 0; l < 4; l++) e[l] = ((w[0] >> (8 * l)) & 0xFFu) | ((qh << (8 - 2 * l)) & 0x300u);
                o.sign = sg[0];
            }
        } else if constexpr (FMT == T_IQ1_S) {       // src/quant/quant_ref.cpp:227-245
            uint32_t w[1];
            words_a2<1>(b + 2 + 4 * s, w);
            const uint32_t qh = s_u16(b + 34 + 2 * s);
            o.a[0] = o.a[1] = __fmul_rn(s_f16(b), (float)(2 * (int)((qh >> 12) & 7u) + 1));
#pragma unroll
            for (int l = 0; l < 4; l++) {
                e[l] = ((w[0] >> (8 * l)) & 0xFFu) | (((qh >> (3 * l)) & 7u) << 8);
                o.off[l] = (qh & 0x8000u) ? -1.125f : -0.875f;
            }
        } else {                                     // IQ1_M, src/quant/quant_ref.cpp:247-283
            uint32_t w[1], sw[2];
            words_a2<1>(b + 4 * s, w);
            words_a2<2>(b + 48, sw);
            const uint32_t qh = s_u16(b + 32 + 2 * s);
            const uint32_t su = ((sw[0] >> 12) & 0xFu) | ((sw[0] >> 24) & 0xF0u) | ((sw[1] >> 4) & 0xF00u) | ((sw[1] >> 16) & 0xF000u);
            const float d = __half2float(__ushort_as_half((unsigned short)su));
            const uint32_t t = (s >= 4 ? sw[1] : sw[0]) >> (16 * ((s >> 1) & 1) + 6 * (s & 1));
            o.a[0] = __fmul_rn(d, (float)(2 * (int)(t & 7u) + 1));
            o.a[1] = __fmul_rn(d, (float)(2 * (int)((t >> 3) & 7u) + 1));
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const uint32_t hn = (qh >> (4 * l)) & 0xFu;
                e[l] = ((w[0] >> (8 * l)) & 0xFFu) | ((hn & 7u) << 8);
                o.off[l] = (hn & 8u) ? -1.125f : -0.875f;
            }
        }
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const uint2 v = *(const uint2*)(tab + e[l] * (2 * G.copies));
            o.u[2 * l] = v.x;
            o.u[2 * l + 1] = v.y;
        }
    }
}

// this lane's copy of the grid table
template <int FMT>
__device__ __forceinline__ const uint32_t* grid_copy(const uint32_t* tab, int lane) {
    constexpr GridTable G = grid_table(FMT);
    return tab + (G.entries ? (lane & (G.copies - 1)) * G.words : 0);
}

// weight k of the sub-block as fp32, its sign not applied yet (FORM_MAGNITUDE)
template <int FMT>
__device__ __forceinline__ float sub32_value(const Sub32& o, int k) {
    const float f = __uint_as_float(prmt(o.u[k >> 2], 0x47000000u, 0x7404u | ((uint32_t)(k & 3) << 4)));   // 2^15 + u
    if (expand_form(FMT) == FORM_AFFINE) return fmaf(o.a[k >> 4], __fsub_rn(f, 32768.0f), -o.c[k >> 4]);
    if (expand_form(FMT) == FORM_OFFSET) return __fmul_rn(o.a[k >> 4], __fadd_rn(f, o.off[k >> 3] - 32768.0f));
    return __fmul_rn(o.a[k >> 4], __fsub_rn(f, 32768.0f));
}
// weights 2 j and 2 j + 1, rounded once to the 16-bit type and packed
template <int FMT, bool F16>
__device__ __forceinline__ uint32_t sub32_pair(const Sub32& o, int j) {
    const float x = sub32_value<FMT>(o, 2 * j), y = sub32_value<FMT>(o, 2 * j + 1);
    uint32_t v;
    if (F16) { const __half2 h = __floats2half2_rn(x, y); v = *(const uint32_t*)&h; }
    else { const __nv_bfloat162 h = __floats2bfloat162_rn(x, y); v = *(const uint32_t*)&h; }
    if (expand_form(FMT) == FORM_MAGNITUDE) {
        // sign bits 2 i and 2 i + 1 of the byte of eight go to bits 15 and 31 (the two shifted copies of the byte never overlap)
        constexpr uint32_t SPREAD[4] = {0x40008000u, 0x10002000u, 0x04000800u, 0x01000200u};
        const uint32_t s8 = (o.sign >> (8 * (j >> 2))) & 0xFFu;
        v ^= (s8 * SPREAD[j & 3]) & 0x80008000u;
    }
    return v;
}

}  // namespace q38b
