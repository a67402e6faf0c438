// q38b_decode1n.cuh -- the granules of q38b_decode1.cuh for several columns: a granule is decoded ONCE into signed int8
// words and integer scales (decode) and multiplied with each column's activations (apply).
//
// Per column the integer sums and the float operations on them are the ones of Gran<FMT>::dot, so a column's result is the
// one-column kernel's, bit for bit.  Where Gran forms P - 2 N (sum of magnitudes minus twice the negative ones) with two
// dp4a per word, the words here carry their signs: three more operations once, one dp4a per word and column.
#pragma once
#include "q38b_decode1.cuh"

namespace q38b {

// 32 weights in the order of the staged activations; s[h]: integer scale of half h
struct Words32 { uint32_t w[8]; int s[2]; float d; };

Q38B_HD int words32_sum(const Words32& g, const uint32_t (&q)[8]) {
    int s0 = 0, s1 = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) { s0 = dp4a_ss(g.w[i], q[i], s0); s1 = dp4a_ss(g.w[4 + i], q[4 + i], s1); }
    return g.s[0] * s0 + g.s[1] * s1;
}

template <int FMT> struct GranN;

// the i-quants with one float factor: fp16 d * dx [* 0.125] * integer sum
template <int FMT> struct GranNWords {
    using W = Words32;
    static constexpr bool EIGHTH = FMT == T_IQ2_XXS || FMT == T_IQ2_XS || FMT == T_IQ2_S || FMT == T_IQ1_S || FMT == T_IQ1_M;
    template <bool A32>
    static Q38B_HD float apply(const W& g, const typename Gran<FMT>::Acts& a) {
        const float f = (float)words32_sum(g, a.q);
        return EIGHTH ? g.d * a.dx * 0.125f * f : g.d * a.dx * f;
    }
};

template <> struct GranN<T_IQ3_XXS> : GranNWords<T_IQ3_XXS> {
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        W g;
        const SP p = row + 98 * (lane >> 3);
        const int s = lane & 7;
        const SP ip = p + (2 + 8 * s);
        const uint32_t aux = sp_ld16(p, 66 + 4 * s) | (sp_ld16(p, 68 + 4 * s) << 16);
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const uint32_t c128 = (l == 0 ? (aux << 7) : (aux >> (7 * l - 7))) & 0x3F80u;
            uint32_t m_lo, m_hi;
            sp_ld64(cb.sign_base + (int)c128, 0, m_lo, m_hi);
            g.w[2 * l] = negate_bytes(cb1(cb, sp_ld8(ip, 2 * l) * 128u), m_lo);
            g.w[2 * l + 1] = negate_bytes(cb1(cb, sp_ld8(ip, 2 * l + 1) * 128u), m_hi);
        }
        g.s[0] = g.s[1] = (int)(2u * (aux >> 28) + 1u);
        g.d = fp16_bits_to_float(sp_ld16(p, 0));
        return g;
    }
};

template <> struct GranN<T_IQ3_S> : GranNWords<T_IQ3_S> {
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        W g;
        const SP p = row + 110 * (lane >> 3);
        const int s = lane & 7;
        uint32_t iw[2];
        sp_ld8b_a2(p + (2 + 8 * s), sp_low2(p) ^ 2u, iw[0], iw[1]);
        const uint32_t qh = sp_ld8(p, 66 + s) << 14;
        const uint32_t sg = sp_ld16(p, 74 + 4 * s) | (sp_ld16(p, 76 + 4 * s) << 16);
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const uint32_t sb = sg >> (8 * l), w = iw[l >> 1];
            g.w[2 * l] = negate_bytes(cb1(cb, byte_x64(w, 2 * (l & 1)) | ((qh >> (2 * l)) & 0x4000u)), sign_mask4(sb & 0xFu));
            g.w[2 * l + 1] = negate_bytes(cb1(cb, byte_x64(w, 2 * (l & 1) + 1) | ((qh >> (2 * l + 1)) & 0x4000u)), sign_mask4((sb >> 4) & 0xFu));
        }
        g.s[0] = g.s[1] = (int)(2u * ((sp_ld8(p, 106 + (s >> 1)) >> (4 * (s & 1))) & 0xFu) + 1u);
        g.d = fp16_bits_to_float(sp_ld16(p, 0));
        return g;
    }
};

template <> struct GranN<T_IQ4_XS> : GranNWords<T_IQ4_XS> {
    static Q38B_HD uint32_t levels(uint32_t nibbles) {   // one of the two look-ups is zero in every byte; -n as int8 for n <= 127
        using U = Unit<T_IQ4_XS>;
        return prmt(U::HR0, U::HR1, ~nibbles) | ((0x80808080u - prmt(U::NL0, U::NL1, nibbles)) ^ 0x80808080u);
    }
    static Q38B_HD W decode(SP row, const Codebook1&, int lane) {
        W g;
        const SP p = row + 136 * (lane >> 3);
        const int s = lane & 7;
        uint32_t w[4];
        sp_ld64(p, 8 + 16 * s, w[0], w[1]);
        sp_ld64(p, 16 + 16 * s, w[2], w[3]);
#pragma unroll
        for (int t = 0; t < 4; t++) { g.w[2 * t] = levels(w[t]); g.w[2 * t + 1] = levels(w[t] >> 16); }
        const uint32_t hdr = sp_ld32(p, 0), sl = sp_ld8(p, 4 + (s >> 1));
        g.s[0] = g.s[1] = (int)(((sl >> (4 * (s & 1))) & 0xFu) | ((((hdr >> 16) >> (2 * s)) & 3u) << 4)) - 32;
        g.d = fp16_bits_to_float(hdr & 0xFFFFu);
        return g;
    }
};

template <> struct GranN<T_Q8_0> : GranNWords<T_Q8_0> {
    static Q38B_HD W decode(SP row, const Codebook1&, int lane) {
        W g;
        const SP p = row + 34 * lane;
        const uint32_t mis = sp_low2(p) ^ 2u;
        const SP wbase = p + 2 - (int)mis;
        uint32_t prev = sp_ld32(wbase, 0);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t next = sp_ld32(wbase, 4 * i + 4);
            g.w[i] = funnel_r(prev, next, mis * 8);
            prev = next;
        }
        g.s[0] = g.s[1] = 1;
        g.d = fp16_bits_to_float(sp_ld16(p, 0));
        return g;
    }
};

Q38B_HD void iq2_words(uint32_t code, uint32_t sign8, uint32_t& w0, uint32_t& w1) {
    w0 = negate_bytes(iq2_bytes(code & 0xFFu), sign_mask4(sign8 & 0xFu));
    w1 = negate_bytes(iq2_bytes(code >> 8), sign_mask4(sign8 >> 4));
}

template <> struct GranN<T_IQ2_XXS> : GranNWords<T_IQ2_XXS> {
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        W g;
        const SP p = row + 66 * (lane >> 3);
        uint32_t a0, a1;
        sp_ld8b_a2(p + (2 + 8 * (lane & 7)), sp_low2(p) ^ 2u, a0, a1);
#pragma unroll
        for (int l = 0; l < 4; l++) iq2_words(code16(cb, (a0 >> (8 * l)) & 0xFFu), ksign_byte((a1 >> (7 * l)) & 127u), g.w[2 * l], g.w[2 * l + 1]);
        g.s[0] = g.s[1] = (int)(2u * (a1 >> 28) + 1u);
        g.d = fp16_bits_to_float(sp_ld16(p, 0));
        return g;
    }
};

template <> struct GranN<T_IQ2_XS> : GranNWords<T_IQ2_XS> {
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        W g;
        const SP p = row + 74 * (lane >> 3);
        const int ib = lane & 7;
        uint32_t w[2];
        sp_ld8b_a2(p + (2 + 8 * ib), sp_low2(p) ^ 2u, w[0], w[1]);
        const uint32_t sc = sp_ld8(p, 66 + ib);
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const uint32_t qv = (w[l >> 1] >> (16 * (l & 1))) & 0xFFFFu;
            iq2_words(code16(cb, qv & 511u), ksign_byte(qv >> 9), g.w[2 * l], g.w[2 * l + 1]);
        }
        g.s[0] = (int)(2u * (sc & 0xFu) + 1u);
        g.s[1] = (int)(2u * (sc >> 4) + 1u);
        g.d = fp16_bits_to_float(sp_ld16(p, 0));
        return g;
    }
};

template <> struct GranN<T_IQ2_S> : GranNWords<T_IQ2_S> {
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        W g;
        const SP p = row + 82 * (lane >> 3);
        const int ib = lane & 7;
        const uint32_t qs = sp_ld16(p, 2 + 4 * ib) | (sp_ld16(p, 4 + 4 * ib) << 16);
        const uint32_t sg = sp_ld16(p, 34 + 4 * ib) | (sp_ld16(p, 36 + 4 * ib) << 16);
        const uint32_t qh = sp_ld8(p, 66 + ib), sc = sp_ld8(p, 74 + ib);
#pragma unroll
        for (int l = 0; l < 4; l++)
            iq2_words(code16(cb, ((qs >> (8 * l)) & 0xFFu) | ((qh << (8 - 2 * l)) & 0x300u)), (sg >> (8 * l)) & 0xFFu, g.w[2 * l], g.w[2 * l + 1]);
        g.s[0] = (int)(2u * (sc & 0xFu) + 1u);
        g.s[1] = (int)(2u * (sc >> 4) + 1u);
        g.d = fp16_bits_to_float(sp_ld16(p, 0));
        return g;
    }
};

template <> struct GranN<T_IQ1_S> : GranNWords<T_IQ1_S> {
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        W g;
        const SP p = row + 50 * (lane >> 3);
        const int ib = lane & 7;
        const uint32_t qs = sp_ld16(p, 2 + 4 * ib) | (sp_ld16(p, 4 + 4 * ib) << 16);
        const uint32_t qh = sp_ld16(p, 34 + 2 * ib);
        const bool minus = (qh & 0x8000u) != 0;
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const uint32_t code = code16(cb, ((qs >> (8 * l)) & 0xFFu) | (((qh >> (3 * l)) & 7u) << 8));
            g.w[2 * l] = iq1_bytes(code & 0xFFu, minus);
            g.w[2 * l + 1] = iq1_bytes(code >> 8, minus);
        }
        g.s[0] = g.s[1] = (int)(2u * ((qh >> 12) & 7u) + 1u);
        g.d = fp16_bits_to_float(sp_ld16(p, 0));
        return g;
    }
};

template <> struct GranN<T_IQ1_M> : GranNWords<T_IQ1_M> {
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        W g;
        const SP p = row + 56 * (lane >> 3);
        const int ib = lane & 7;
        const uint32_t qs = sp_ld16(p, 4 * ib) | (sp_ld16(p, 4 * ib + 2) << 16);
        const uint32_t qh = sp_ld16(p, 32 + 2 * ib);
        const uint32_t s0 = sp_ld16(p, 48), s1 = sp_ld16(p, 50), s2 = sp_ld16(p, 52), s3 = sp_ld16(p, 54);
        const uint32_t su = (s0 >> 12) | ((s1 >> 8) & 0x00F0u) | ((s2 >> 4) & 0x0F00u) | (s3 & 0xF000u);
        const uint32_t scw = (ib >> 1) == 0 ? s0 : (ib >> 1) == 1 ? s1 : (ib >> 1) == 2 ? s2 : s3;
        const uint32_t t = scw >> (6 * (ib & 1));
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const uint32_t hn = (qh >> (4 * l)) & 0xFu;
            const uint32_t code = code16(cb, ((qs >> (8 * l)) & 0xFFu) | ((hn & 7u) << 8));
            const bool minus = (hn & 8u) != 0;
            g.w[2 * l] = iq1_bytes(code & 0xFFu, minus);
            g.w[2 * l + 1] = iq1_bytes(code >> 8, minus);
        }
        g.s[0] = (int)(2u * (t & 7u) + 1u);
        g.s[1] = (int)(2u * ((t >> 3) & 7u) + 1u);
        g.d = fp16_bits_to_float(su);
        return g;
    }
};

template <> struct GranN<T_Q2_K> {
    struct W { uint32_t w[8]; uint32_t sc; float d, dmin; };
    static Q38B_HD W decode(SP row, const Codebook1&, int lane) {
        W g;
        const SP p = row + 84 * (lane >> 3);
        const int ib = lane & 7, n = ib >> 2, j = ib & 3;
#pragma unroll
        for (int i = 0; i < 8; i++) g.w[i] = (sp_ld32(p, 16 + 32 * n + 4 * i) >> (2 * j)) & 0x03030303u;
        g.sc = sp_ld16(p, 2 * ib);
        const uint32_t dd = sp_ld32(p, 80);
        g.d = fp16_bits_to_float(dd & 0xFFFFu);
        g.dmin = fp16_bits_to_float(dd >> 16);
        return g;
    }
    template <bool A32>
    static Q38B_HD float apply(const W& g, const Gran<T_Q2_K>::Acts& a) {
        int S0 = 0, S1 = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) { S0 = dp4a_us(g.w[i], a.q[i], S0); S1 = dp4a_us(g.w[4 + i], a.q[4 + i], S1); }
        const int sumi = (int)(g.sc & 0xFu) * S0 + (int)((g.sc >> 8) & 0xFu) * S1;
        const int msum = (int)((g.sc >> 4) & 0xFu) * a.bs0 + (int)(g.sc >> 12) * a.bs1;
        return g.d * a.dx * (float)sumi - g.dmin * a.dx * (float)msum;
    }
};

template <int NBITS> struct GranNQ45K {
    using One = GranQ45K<NBITS>;
    struct W { uint32_t lo[8], hi[8]; int sc0, sc1, mn0, mn1; float d, dmin; };
    static Q38B_HD W decode(SP row, const Codebook1&, int lane) {
        W g;
        const int pr = lane & 15, pp = pr & 3;
        const SP p = row + One::BB * (pr >> 2);
        uint32_t v0[4], v1[4], hd[4];
        sp_ld128(p, One::QS + 32 * pp, v0);
        sp_ld128(p, One::QS + 32 * pp + 16, v1);
        sp_ld128(p, 0, hd);
        const uint32_t dd = hd[0], u0 = hd[1], u1 = hd[2], u2 = hd[3];
        const bool hi_half = pp >= 2;
        const uint32_t sc4 = hi_half ? ((u2 & 0x0F0F0F0Fu) | ((u0 >> 2) & 0x30303030u)) : (u0 & 0x3F3F3F3Fu);
        const uint32_t mn4 = hi_half ? (((u2 >> 4) & 0x0F0F0F0Fu) | ((u1 >> 2) & 0x30303030u)) : (u1 & 0x3F3F3F3Fu);
        const uint32_t sh = 16u * (uint32_t)(pp & 1);
        g.sc0 = (int)((sc4 >> sh) & 0xFFu); g.sc1 = (int)((sc4 >> (sh + 8)) & 0xFFu);
        g.mn0 = (int)((mn4 >> sh) & 0xFFu); g.mn1 = (int)((mn4 >> (sh + 8)) & 0xFFu);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t w = i < 4 ? v0[i & 3] : v1[i & 3];
            g.lo[i] = w & 0x0F0F0F0Fu;
            g.hi[i] = (w >> 4) & 0x0F0F0F0Fu;
        }
        if (NBITS == 5) {
            uint32_t h0[4], h1[4];
            sp_ld128(p, 16, h0);
            sp_ld128(p, 32, h1);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t hb = (i < 4 ? h0[i & 3] : h1[i & 3]) >> (2u * (uint32_t)pp);
                g.lo[i] |= (hb << 4) & 0x10101010u;
                g.hi[i] |= (hb << 3) & 0x10101010u;
            }
        }
        g.d = fp16_bits_to_float(dd & 0xFFFFu);
        g.dmin = fp16_bits_to_float(dd >> 16);
        return g;
    }
    template <bool A32>
    static Q38B_HD float apply(const W& g, const typename One::Acts& a) {
        int lo = 0, hi = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) { lo = dp4a_ss(g.lo[i], a.q[i], lo); hi = dp4a_ss(g.hi[i], a.q[8 + i], hi); }
        if (A32)
            return g.d * (a.dx * (float)(g.sc0 * lo) + a.dx1 * (float)(g.sc1 * hi)) - g.dmin * (a.dx * (float)(g.mn0 * a.bs0) + a.dx1 * (float)(g.mn1 * a.bs1));
        const int sumi = g.sc0 * lo + g.sc1 * hi;
        const int msum = g.mn0 * a.bs0 + g.mn1 * a.bs1;
        return g.d * a.dx * (float)sumi - g.dmin * a.dx * (float)msum;
    }
};
template <> struct GranN<T_Q4_K> : GranNQ45K<4> {};
template <> struct GranN<T_Q5_K> : GranNQ45K<5> {};

template <> struct GranN<T_Q6_K> {
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
        if (A32) {
            float acc = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) acc += a.dxs[j] * (float)(g.sc[j] * d4[j]);
            return g.d * acc;
        }
        int sumi = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) sumi += g.sc[j] * d4[j];
        return g.d * a.dx * (float)sumi;
    }
};

}  // namespace q38b
