// q38b_decode1n.cuh -- variants of the granules of q38b_decode1.cuh: IQ2 / IQ1 with expanded grid tables (one column), and the
// several-column granule of Q6_K with per-32 activations.
#pragma once
#include "q38b_decode1.cuh"

namespace q38b {

// ---------------------------------------------------------------------------------------------------------------
// IQ2_XXS, IQ2_XS, IQ2_S, IQ1_S, IQ1_M with the whole shared memory of an SM: the grid as eight bytes an entry (the
// magnitudes 8, 25, 43; for IQ1 eight times the level number 0, 1, 2), in as many copies as fit 64 KB, so that one 64-bit
// load replaces a 16-bit code, its expansion to two PRMT selectors and two PRMT; lane l reads copy l % copies (16 copies:
// a half warp meets no bank).  The seven-bit sign codes of IQ2_XXS / IQ2_XS come as byte masks from the table IQ3_XXS has.
// The integer sums are Gran<FMT>'s, which serves rows too long for these tables and the plans with two CTAs an SM.  Measured with one column, 19456 x 2816
// IQ2_XXS: 17.8 -> 13.7 us; 2816 x 9728 IQ2_S 10.9 -> 8.5 us.
// ---------------------------------------------------------------------------------------------------------------
Q38B_HD constexpr int gridx_copies(int fmt) { return fmt == T_IQ2_XXS || fmt == T_IQ2_XS ? 16 : fmt == T_IQ2_S ? 8 : fmt == T_IQ1_S || fmt == T_IQ1_M ? 4 : 0; }
Q38B_HD constexpr int gridx_bytes(int fmt) { return code16_entries(fmt) * gridx_copies(fmt) * 8; }
Q38B_HD constexpr bool gridx_signs(int fmt) { return fmt == T_IQ2_XXS || fmt == T_IQ2_XS; }
// bytes 0..3 and 4..7 of the entry with 16-bit code `code`
template <int FMT>
Q38B_HD void gridx_entry(uint32_t code, uint32_t& lo, uint32_t& hi) {
    constexpr uint32_t LEVELS = FMT == T_IQ1_S || FMT == T_IQ1_M ? 0x00100800u : 0x002B1908u;
    lo = prmt(LEVELS, 0u, sel_from_codes(code & 0xFFu));
    hi = prmt(LEVELS, 0u, sel_from_codes(code >> 8));
}

// A granule as looked up: grid bytes g, sign masks m (IQ2), delta of each group of eight (IQ1: the weight is g + c)
struct RawGran { uint32_t g[8], m[8]; int c[4]; int s[2]; };
template <int FMT> struct GranX {
    static constexpr bool IQ1 = FMT == T_IQ1_S || FMT == T_IQ1_M;
    static constexpr int STRIDE = 8 * gridx_copies(FMT), STRIDE_LOG2 = gridx_copies(FMT) == 16 ? 7 : gridx_copies(FMT) == 8 ? 6 : 5;
    struct Acts : Gran<FMT>::Acts { int bs[IQ1 ? 4 : 1]; };   // bs: sums of eight activations
    template <bool A32>
    static Q38B_HD void load_acts(Acts& a, SP aq, SP ad, int lane) {
        Gran<FMT>::template load_acts<A32>(a, aq, ad, lane);
        if (IQ1) {
#pragma unroll
            for (int l = 0; l < 4; l++) a.bs[IQ1 ? l : 0] = dp4a_ss(0x01010101u, a.q[2 * l], dp4a_ss(0x01010101u, a.q[2 * l + 1], 0));
        }
    }
    static Q38B_HD void entry(const Codebook1& cb, uint32_t e_times_stride, uint32_t& lo, uint32_t& hi) { sp_ld64(cb.lane_base + (int)e_times_stride, 0, lo, hi); }
    // bits [at, at + n) of w, times the entry stride
    static Q38B_HD uint32_t index(uint32_t w, int at, int n) {
        const uint32_t mask = ((1u << n) - 1u) << STRIDE_LOG2;
        return (at >= STRIDE_LOG2 ? (w >> (at - STRIDE_LOG2)) : (w << (STRIDE_LOG2 - at))) & mask;
    }
    static Q38B_HD void look_up(SP row, const Codebook1& cb, int lane, RawGran& o) {
        const SP p = row + Unit<FMT>::BLOCK_BYTES * (lane >> 3);
        const int ib = lane & 7;
        if constexpr (FMT == T_IQ2_XXS) {
            uint32_t a0, a1;
            sp_ld8b_a2(p + (2 + 8 * ib), sp_low2(p) ^ 2u, a0, a1);
#pragma unroll
            for (int l = 0; l < 4; l++) {
                entry(cb, index(a0, 8 * l, 8), o.g[2 * l], o.g[2 * l + 1]);
                sp_ld64(cb.sign_base + (int)((l == 0 ? (a1 << 7) : (a1 >> (7 * l - 7))) & 0x3F80u), 0, o.m[2 * l], o.m[2 * l + 1]);
            }
            o.s[0] = o.s[1] = (int)(2u * (a1 >> 28) + 1u);
        } else if constexpr (FMT == T_IQ2_XS) {
            uint32_t w[2];
            sp_ld8b_a2(p + (2 + 8 * ib), sp_low2(p) ^ 2u, w[0], w[1]);
            const uint32_t sc = sp_ld8(p, 66 + ib);
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const int at = 16 * (l & 1);
                entry(cb, index(w[l >> 1], at, 9), o.g[2 * l], o.g[2 * l + 1]);
                sp_ld64(cb.sign_base + (int)((w[l >> 1] >> (at + 2)) & 0x3F80u), 0, o.m[2 * l], o.m[2 * l + 1]);
            }
            o.s[0] = (int)(2u * (sc & 0xFu) + 1u);
            o.s[1] = (int)(2u * (sc >> 4) + 1u);
        } else if constexpr (FMT == T_IQ2_S) {
            const uint32_t qs = sp_ld16(p, 2 + 4 * ib) | (sp_ld16(p, 4 + 4 * ib) << 16);
            const uint32_t sg = sp_ld16(p, 34 + 4 * ib) | (sp_ld16(p, 36 + 4 * ib) << 16);
            const uint32_t qh = sp_ld8(p, 66 + ib), sc = sp_ld8(p, 74 + ib);
#pragma unroll
            for (int l = 0; l < 4; l++) {
                entry(cb, index(qs, 8 * l, 8) | ((qh << (8 - 2 * l + STRIDE_LOG2)) & (0x300u << STRIDE_LOG2)), o.g[2 * l], o.g[2 * l + 1]);
                o.m[2 * l] = sign_mask4((sg >> (8 * l)) & 0xFu);
                o.m[2 * l + 1] = sign_mask4((sg >> (8 * l + 4)) & 0xFu);
            }
            o.s[0] = (int)(2u * (sc & 0xFu) + 1u);
            o.s[1] = (int)(2u * (sc >> 4) + 1u);
        } else if constexpr (FMT == T_IQ1_S) {
            const uint32_t qs = sp_ld16(p, 2 + 4 * ib) | (sp_ld16(p, 4 + 4 * ib) << 16);
            const uint32_t qh = sp_ld16(p, 34 + 2 * ib);
#pragma unroll
            for (int l = 0; l < 4; l++) {
                entry(cb, index(qs, 8 * l, 8) | (((qh >> (3 * l)) & 7u) << (8 + STRIDE_LOG2)), o.g[2 * l], o.g[2 * l + 1]);
                o.c[l] = (qh & 0x8000u) ? -9 : -7;   // 8 (level - 1) + 1, or - 1
            }
            o.s[0] = o.s[1] = (int)(2u * ((qh >> 12) & 7u) + 1u);
        } else {
            const uint32_t qs = sp_ld16(p, 4 * ib) | (sp_ld16(p, 4 * ib + 2) << 16);
            const uint32_t qh = sp_ld16(p, 32 + 2 * ib);
            const uint32_t s0 = sp_ld16(p, 48), s1 = sp_ld16(p, 50), s2 = sp_ld16(p, 52), s3 = sp_ld16(p, 54);
            const uint32_t t = ((ib >> 1) == 0 ? s0 : (ib >> 1) == 1 ? s1 : (ib >> 1) == 2 ? s2 : s3) >> (6 * (ib & 1));
#pragma unroll
            for (int l = 0; l < 4; l++) {
                const uint32_t hn = qh >> (4 * l);
                entry(cb, index(qs, 8 * l, 8) | ((hn & 7u) << (8 + STRIDE_LOG2)), o.g[2 * l], o.g[2 * l + 1]);
                o.c[l] = (hn & 8u) ? -9 : -7;
            }
            o.s[0] = (int)(2u * (t & 7u) + 1u);
            o.s[1] = (int)(2u * ((t >> 3) & 7u) + 1u);
        }
    }
    static Q38B_HD void block_scale(SP block, float& d, float& m) { Gran<FMT>::block_scale(block, d, m); }
    // P - 2 N (IQ2) or P + c * (sum of the group's activations) (IQ1)
    static Q38B_HD int idot(SP row, const Acts& a, const Codebook1& cb, int lane, int& msum) {
        RawGran o;
        look_up(row, cb, lane, o);
        msum = 0;
        int S[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int P = 0, N = 0;
#pragma unroll
            for (int i = 4 * h; i < 4 * h + 4; i++) {
                P = dp4a_us(o.g[i], a.q[i], P);
                if (!IQ1) N = dp4a_us(o.g[i] & o.m[i], a.q[i], N);
            }
            S[h] = IQ1 ? P + o.c[2 * h] * a.bs[0 + (IQ1 ? 2 * h : 0)] + o.c[2 * h + 1] * a.bs[IQ1 ? 2 * h + 1 : 0] : P - 2 * N;
        }
        return o.s[0] * S[0] + o.s[1] * S[1];
    }
    template <bool A32>
    static Q38B_HD float dot(SP row, const Acts& a, const Codebook1& cb, int lane) {
        int ms;
        const int sum = idot(row, a, cb, lane, ms);
        return gran_value<Gran<FMT>, FMT>(row + Unit<FMT>::BLOCK_BYTES * (lane >> 3), a.dx, sum, ms);
    }
};

// Several columns of Q6_K with per-32 activations: a granule is decoded ONCE into signed int8 words and integer scales (decode)
// and multiplied with each column's activations (apply), whose result is Gran<T_Q6_K>::dot<true>'s, bit for bit.  (Its granules
// take eight weights of each of four sub-blocks, which the fragments of q38b_decode.cuh cannot add up in the same order.)
template <int FMT> struct GranN;
template <> struct GranN<T_Q6_K> {
    using Acts = Gran<T_Q6_K>::Acts;
    template <bool A32>
    static Q38B_HD void load_acts(Acts& a, SP aq, SP ad, int lane) { Gran<T_Q6_K>::load_acts<A32>(a, aq, ad, lane); }
    struct W { uint32_t w[8]; int sc[4]; float d; };
    static Q38B_HD W decode(SP row, const Codebook1&, int lane) {
        W g;
        const int n = (lane >> 2) & 1, i = lane & 3;
        const SP p = row + 210 * (lane >> 3);
        const uint32_t mis = sp_low2(p);
        uint32_t qa[2], qb[2], qh[2];
        sp_ld8b_a2(p + (64 * n + 8 * i), mis, qa[0], qa[1]);
        sp_ld8b_a2(p + (64 * n + 32 + 8 * i), mis, qb[0], qb[1]);
        sp_ld8b_a2(p + (128 + 32 * n + 8 * i), mis, qh[0], qh[1]);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            g.w[k] = Unit<T_Q6_K>::q6(qa[k], qh[k] << 4);
            g.w[2 + k] = Unit<T_Q6_K>::q6(qb[k], qh[k] << 2);
            g.w[4 + k] = Unit<T_Q6_K>::q6(qa[k] >> 4, qh[k]);
            g.w[6 + k] = Unit<T_Q6_K>::q6(qb[k] >> 4, qh[k] >> 2);
        }
        const SP sc = p + (192 + 8 * n + (i >> 1));
#pragma unroll
        for (int j = 0; j < 4; j++) g.sc[j] = sp_ld8s(sc, 2 * j);
        g.d = fp16_bits_to_float(sp_ld16(p, 208));
        return g;
    }
    template <bool A32>
    static Q38B_HD float apply(const W& g, const Gran<T_Q6_K>::Acts& a) {
        int d4[4];
#pragma unroll
        for (int j = 0; j < 4; j++) d4[j] = dp4a_ss(g.w[2 * j + 1], a.q[2 * j + 1], dp4a_ss(g.w[2 * j], a.q[2 * j], 0));
        static_assert(A32, "Q8_K columns run on the several-column kernel");
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) acc += a.dxs[j] * (float)(g.sc[j] * d4[j]);
        return g.d * acc;
    }
};

}  // namespace q38b
