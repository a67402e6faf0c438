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
            const uint32_t t = sp_ld16(p, 48 + 2 * (ib >> 1)) >> (6 * (ib & 1));
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

// ---------------------------------------------------------------------------------------------------------------
// Two to four columns on the one-column kernel: a granule is decoded ONCE into signed int8 words and integer scales (decode) and
// multiplied with each column's activations.  isum<> is Gran<FMT>::idot's integer, apply<A32> Gran<FMT>::dot's float: a column's
// result is the one-column launch's, bit for bit.  Where Gran forms P - 2 N (sum of magnitudes minus twice the negative ones) with
// two dp4a per word, the words here carry their signs: three more operations once, one dp4a per word and column.
// ---------------------------------------------------------------------------------------------------------------
// 32 weights in the order of the staged activations; s[h]: integer scale of half h
struct Words32 { uint32_t w[8]; int s[2]; };

template <int FMT> struct GranN;

// the formats with one float factor: fp16 d * dx * integer sum
template <int FMT> struct GranNWords {
    using W = Words32;
    using Acts = typename Gran<FMT>::Acts;
    template <bool A32>
    static Q38B_HD void load_acts(Acts& a, SP aq, SP ad, int lane) { Gran<FMT>::template load_acts<A32>(a, aq, ad, lane); }
    static Q38B_HD void block_scale(SP block, float& d, float& m) { Gran<FMT>::block_scale(block, d, m); }
    static Q38B_HD int isum(const W& g, const Acts& a, int& msum) {
        int s0 = 0, s1 = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) { s0 = dp4a_ss(g.w[i], a.q[i], s0); s1 = dp4a_ss(g.w[4 + i], a.q[4 + i], s1); }
        msum = 0;
        return g.s[0] * s0 + g.s[1] * s1;
    }
    // d: the block's factor (block_scale)
    template <bool A32>
    static Q38B_HD float apply(const W& g, const Acts& a, float d, float) {
        int ms;
        const int sum = isum(g, a, ms);
        return block_value(d * a.dx * Unit<FMT>::FACTOR, sum);
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
        return g;
    }
};

template <> struct GranN<T_Q8_0> : GranNWords<T_Q8_0> {
    static Q38B_HD void block_scale(SP block, float& d, float& m) { d = fp16_bits_to_float(sp_ld16(block, 0)); m = 0.0f; }   // of a lane's own 34 bytes
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
        return g;
    }
};

// IQ2 / IQ1 with their expanded grids
template <int FMT> struct GranNX : GranNWords<FMT> {
    using X = GranX<FMT>;
    using W = Words32;
    static Q38B_HD W decode(SP row, const Codebook1& cb, int lane) {
        RawGran o;
        X::look_up(row, cb, lane, o);
        W w;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (X::IQ1) w.w[i] = ((o.g[i] | 0x80808080u) - (o.c[i >> 1] == -9 ? 0x09090909u : 0x07070707u)) ^ 0x80808080u;
            else w.w[i] = negate_bytes(o.g[i], o.m[i]);
        }
        w.s[0] = o.s[0];
        w.s[1] = o.s[1];
        return w;
    }
};
template <> struct GranN<T_IQ2_XXS> : GranNX<T_IQ2_XXS> {};
template <> struct GranN<T_IQ2_XS> : GranNX<T_IQ2_XS> {};
template <> struct GranN<T_IQ2_S> : GranNX<T_IQ2_S> {};
template <> struct GranN<T_IQ1_S> : GranNX<T_IQ1_S> {};
template <> struct GranN<T_IQ1_M> : GranNX<T_IQ1_M> {};

template <> struct GranN<T_Q2_K> {
    using Acts = Gran<T_Q2_K>::Acts;
    template <bool A32>
    static Q38B_HD void load_acts(Acts& a, SP aq, SP ad, int lane) { Gran<T_Q2_K>::load_acts<A32>(a, aq, ad, lane); }
    static Q38B_HD void block_scale(SP block, float& d, float& m) { Gran<T_Q2_K>::block_scale(block, d, m); }
    struct W { uint32_t w[8]; uint32_t sc; };
    static Q38B_HD W decode(SP row, const Codebook1&, int lane) {
        W g;
        const SP p = row + 84 * (lane >> 3);
        const int ib = lane & 7, n = ib >> 2, j = ib & 3;
#pragma unroll
        for (int i = 0; i < 8; i++) g.w[i] = (sp_ld32(p, 16 + 32 * n + 4 * i) >> (2 * j)) & 0x03030303u;
        g.sc = sp_ld16(p, 2 * ib);
        return g;
    }
    static Q38B_HD int isum(const W& g, const Acts& a, int& msum) {
        int S0 = 0, S1 = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) { S0 = dp4a_us(g.w[i], a.q[i], S0); S1 = dp4a_us(g.w[4 + i], a.q[4 + i], S1); }
        msum = (int)((g.sc >> 4) & 0xFu) * a.bs0 + (int)(g.sc >> 12) * a.bs1;
        return (int)(g.sc & 0xFu) * S0 + (int)((g.sc >> 8) & 0xFu) * S1;
    }
    template <bool A32>
    static Q38B_HD float apply(const W& g, const Acts& a, float d, float m) {
        int ms;
        const int sum = isum(g, a, ms);
        return block_value_min(d * a.dx, sum, m * a.dx, ms);
    }
};

template <int NBITS> struct GranNQ45K {
    using One = GranQ45K<NBITS>;
    using Acts = typename One::Acts;
    template <bool A32>
    static Q38B_HD void load_acts(Acts& a, SP aq, SP ad, int lane) { One::template load_acts<A32>(a, aq, ad, lane); }
    static Q38B_HD void block_scale(SP block, float& d, float& m) { One::block_scale(block, d, m); }
    struct W { uint32_t lo[8], hi[8]; int sc0, sc1, mn0, mn1; };
    static Q38B_HD W decode(SP row, const Codebook1&, int lane) {
        W g;
        const int pr = lane & 15, pp = pr & 3;
        const SP p = row + One::BB * (pr >> 2);
        uint32_t v0[4], v1[4], hd[4];
        sp_ld128(p, One::QS + 32 * pp, v0);
        sp_ld128(p, One::QS + 32 * pp + 16, v1);
        sp_ld128(p, 0, hd);
        const uint32_t u0 = hd[1], u1 = hd[2], u2 = hd[3];
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
        return g;
    }
    static Q38B_HD void sums(const W& g, const Acts& a, int (&v)[2], int (&m)[2]) {
        int lo = 0, hi = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) { lo = dp4a_ss(g.lo[i], a.q[i], lo); hi = dp4a_ss(g.hi[i], a.q[8 + i], hi); }
        v[0] = g.sc0 * lo; v[1] = g.sc1 * hi;
        m[0] = g.mn0 * a.bs0; m[1] = g.mn1 * a.bs1;
    }
    static Q38B_HD int isum(const W& g, const Acts& a, int& msum) {
        int v[2], m[2];
        sums(g, a, v, m);
        msum = m[0] + m[1];
        return v[0] + v[1];
    }
    template <bool A32>
    static Q38B_HD float apply(const W& g, const Acts& a, float d, float dmin) {
        int v[2], m[2];
        sums(g, a, v, m);
        if (!A32) return block_value_min(d * a.dx, v[0] + v[1], dmin * a.dx, m[0] + m[1]);
        const float kv = fmaf(a.dx1, (float)v[1], fmul_once(a.dx, (float)v[0])), km = fmaf(a.dx1, (float)m[1], fmul_once(a.dx, (float)m[0]));
        return fmaf(-dmin, km, fmul_once(d, kv));
    }
};
template <> struct GranN<T_Q4_K> : GranNQ45K<4> {};
template <> struct GranN<T_Q5_K> : GranNQ45K<5> {};

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
        return g;
    }
};

template <> struct GranN<T_Q6_K> {
    using Acts = Gran<T_Q6_K>::Acts;
    template <bool A32>
    static Q38B_HD void load_acts(Acts& a, SP aq, SP ad, int lane) { Gran<T_Q6_K>::load_acts<A32>(a, aq, ad, lane); }
    static Q38B_HD void block_scale(SP block, float& d, float& m) { Gran<T_Q6_K>::block_scale(block, d, m); }
    struct W { uint32_t w[8]; int sc[4]; };
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
        return g;
    }
    static Q38B_HD void groups(const W& g, const Acts& a, int (&d4)[4]) {
#pragma unroll
        for (int j = 0; j < 4; j++) d4[j] = dp4a_ss(g.w[2 * j + 1], a.q[2 * j + 1], dp4a_ss(g.w[2 * j], a.q[2 * j], 0));
    }
    static Q38B_HD int isum(const W& g, const Acts& a, int& msum) {
        int d4[4], sum = 0;
        groups(g, a, d4);
#pragma unroll
        for (int j = 0; j < 4; j++) sum += g.sc[j] * d4[j];
        msum = 0;
        return sum;
    }
    template <bool A32>
    static Q38B_HD float apply(const W& g, const Acts& a, float d, float) {
        int d4[4];
        groups(g, a, d4);
        if (!A32) {
            int sum = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) sum += g.sc[j] * d4[j];
            return block_value(d * a.dx, sum);
        }
        float acc = 0.0f;   // group j of the granule lies in 32-weight block 4n + j of the super-block
#pragma unroll
        for (int j = 0; j < 4; j++) acc += a.dxs[j] * (float)(g.sc[j] * d4[j]);
        return d * acc;
    }
};

}  // namespace q38b
