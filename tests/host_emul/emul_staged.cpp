// CPU emulation of one consumer warp of the several-column matvec as the kernel runs it on Q8_K columns: sign masks from the
// staged table, minima from the staged sums (two digits), the run of zeros of the formats whose scale changes every 16 weights,
// grids as eight-byte entries.  32 host threads play the lanes; mma and shuffles are rendezvous points that apply the PTX
// fragment layouts.
#include <pthread.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../qwengine_b200/csrc/q38b_decode.cuh"

namespace {
thread_local int tl_lane = 0;
pthread_barrier_t g_bar;
uint32_t g_a[32][4], g_b[32][2], g_sh[32];
}  // namespace

namespace q38b {
int emul_lane() { return tl_lane; }

void emul_mma(int (&c)[4], const uint32_t* a, int n_a, const uint32_t* b, int n_b) {
    memcpy(g_a[tl_lane], a, 4 * (size_t)n_a);
    memcpy(g_b[tl_lane], b, 4 * (size_t)n_b);
    pthread_barrier_wait(&g_bar);
    for (int ci = 0; ci < 4; ci++) {
        const int m = (tl_lane >> 2) + 8 * (ci >> 1), n = 2 * (tl_lane & 3) + (ci & 1);
        for (int k = 0; k < 16 * n_b; k++) {
            // A[m][k]: lane 4 (m % 8) + (k % 16) / 4, register m / 8 + 2 (k / 16); B[k][n]: lane 4 n + (k % 16) / 4, register k / 16
            const int q = (k & 15) >> 2, sh = 8 * (k & 3);
            c[ci] += (int)(int8_t)(g_a[(m & 7) * 4 + q][(m >> 3) + 2 * (k >> 4)] >> sh) * (int)(int8_t)(g_b[n * 4 + q][k >> 4] >> sh);
        }
    }
    pthread_barrier_wait(&g_bar);
}

uint32_t emul_shfl(uint32_t v, int src) {
    g_sh[tl_lane] = v;
    pthread_barrier_wait(&g_bar);
    const uint32_t r = g_sh[src & 31];
    pthread_barrier_wait(&g_bar);
    return r;
}
}  // namespace q38b

#include "../../qwengine_b200/csrc/q38b_decode1n.cuh"
#define Q38B_CODEBOOK_QUALIFIER static const
#include "../../qwengine_b200/csrc/codebooks.inc"

using namespace q38b;

namespace {
struct Job {
    int nsb, nb, slot;
    const int* shift;
    const uint8_t *stage, *actq, *cb, *sgn, *zero, *bsum;
    const float* actd;
    float* y;
};
struct Lane { const Job* job; int lane; };

template <int FMT>
void* run_lane(void* arg) {
    using U = Unit<FMT>;
    const Job& j = *((const Lane*)arg)->job;
    tl_lane = ((const Lane*)arg)->lane;
    const int g = tl_lane >> 2, t = tl_lane & 3;
    constexpr bool Q2 = FMT == T_Q2_K, HALVES = FMT == T_IQ2_XS || FMT == T_IQ2_S || FMT == T_IQ1_M;
    FragEnv e;
    e.t = t;
    e.cb = sp_from(j.cb);
    e.cb_shift = gridx_copies(FMT) > 0 ? 3 : 2;
    e.sgn = sp_from(j.sgn) + 8 * (tl_lane & (SIGN_COPIES - 1));
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int sb = 0; sb < j.nsb; sb++) {
        const SP pA = sp_from(j.stage + (size_t)g * j.slot + j.shift[g] + (size_t)sb * U::BLOCK_BYTES);
        const SP pB = sp_from(j.stage + (size_t)(g + 8) * j.slot + j.shift[g + 8] + (size_t)sb * U::BLOCK_BYTES);
        e.q = sp_from(j.actq + ((size_t)(g < j.nb ? g : 0) * j.nsb + sb) * 256) + U::ACT_STEP * t;
        e.q_half[0] = HALVES && t >= 2 ? sp_from(j.zero) : e.q;
        e.q_half[1] = HALVES && t < 2 ? sp_from(j.zero) : e.q;
        e.bsum = sp_from(j.bsum + ((size_t)sb * 8 + g) * (Q2 ? 32 : 16)) + 4 * t;
        typename U::Row A, B;
        U::row(pA, t, A);
        U::row(pB, t, B);
        int sums[4] = {0, 0, 0, 0}, cm[4] = {0, 0, 0, 0};
        float dA, mA, dB, mB;
        U::dd(pA, A, dA, mA);
        U::dd(pB, B, dB, mB);
        if constexpr (U::HAS_MIN) U::mins(A, B, e, cm);
        for (int h = 0; h < 2; h++)
            U::template half<true>(A, B, pA, pB, h, e, cm, [&](int s, const int (&v)[4]) {
                for (int i = 0; i < 4; i++) {
                    if (U::SCALE32) acc[i] += block_value(U::d32(i < 2 ? pA : pB, s) * j.actd[sb * 8 + 2 * t + (i & 1)], v[i]);
                    else sums[i] += v[i];
                }
            });
        for (int i = 0; i < 4 && !U::SCALE32; i++) {
            const float dx = j.actd[sb * 8 + 2 * t + (i & 1)], d = i < 2 ? dA : dB;
            acc[i] += U::HAS_MIN ? block_value_min(d * dx, sums[i], (i < 2 ? mA : mB) * dx, cm[i]) : block_value(d * dx * U::FACTOR, sums[i]);
        }
    }
    for (int i = 0; i < 4; i++) j.y[(g + 8 * (i >> 1)) * 8 + 2 * t + (i & 1)] = acc[i];
    return nullptr;
}

// the grid as the kernel stages it, one copy
template <int FMT>
void fill_grid(uint8_t* cb, const uint16_t* codes) {
    for (int i = 0; i < code16_entries(FMT); i++) {
        uint32_t w[2];
        gridx_entry<FMT>(codes[i], w[0], w[1]);
        if (FMT == T_IQ1_S || FMT == T_IQ1_M)
            for (uint32_t& v : w) v = ((v | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
        memcpy(cb + 8 * i, w, 8);
    }
}
}  // namespace

// W: 16 packed rows; xq: Q8_K blocks [nb][K / 256]; addr_lo: low address bits of row 0; y: [16][8]
extern "C" int emul_staged_tile(int fmt, int K, const uint8_t* W, const uint8_t* xq, int nb, int addr_lo, float* y) {
    const int bb = block_bytes(fmt) * (fmt == T_Q8_0 && block_bytes(fmt) == 34 ? 8 : 1), nsb = K / 256, row_bytes = nsb * bb;
    if (!bb) return -1;
    const int slot = (row_bytes + 32 + 15) / 16 * 16 + 16;
    std::vector<uint64_t> mem[6];
    auto bytes = [&](int i, size_t n, uint8_t v) {   // 16-byte aligned
        mem[i].assign(n / 8 + 4, 0x0101010101010101ull * v);
        return (uint8_t*)(((uintptr_t)mem[i].data() + 15) & ~(uintptr_t)15);
    };
    uint8_t *st = bytes(0, (size_t)16 * slot + 64, 0xA5), *actq = bytes(1, (size_t)nb * K, 0), *cb = bytes(2, 2048 * 8, 0xA5);
    uint8_t *sgn = bytes(3, 128 * 8 * SIGN_COPIES, 0xA5), *zero = bytes(4, 264, 0), *bsum = bytes(5, (size_t)nsb * 8 * 32, 0xA5);
    int shift[16];
    for (int r = 0; r < 16; r++) {
        shift[r] = (addr_lo + r * row_bytes) & 15;
        memcpy(st + (size_t)r * slot + shift[r], W + (size_t)r * row_bytes, (size_t)row_bytes);
    }
    std::vector<float> actd((size_t)nsb * 8, 0.f);
    const int per = fmt == T_Q2_K ? 16 : 32, n_sub = 256 / per;
    for (int c = 0; c < nb; c++)
        for (int sb = 0; sb < nsb; sb++) {
            const uint8_t* blk = xq + ((size_t)c * nsb + sb) * 292;
            memcpy(&actd[(size_t)sb * 8 + c], blk, 4);
            for (int k = 0; k < 256; k++) actq[((size_t)c * nsb + sb) * 256 + (k & ~31) + act_stage_pos(fmt, k & 31)] = blk[4 + k];
            for (int s = 0; s < n_sub; s++) {
                int sum = 0;
                for (int k = 0; k < per; k++) sum += (int8_t)blk[4 + s * per + k];
                uint8_t* to = bsum + ((size_t)sb * 8 + c) * 2 * n_sub;
                to[s] = (uint8_t)(sum & 63);
                to[n_sub + s] = (uint8_t)(sum >> 6);
            }
        }
    for (int i = 0; i < 128 * SIGN_COPIES; i++) {
        uint32_t m[2];
        sign_masks7((uint32_t)i / SIGN_COPIES, m[0], m[1]);
        memcpy(sgn + 8 * i, m, 8);
    }
    void* (*lane)(void*) = nullptr;
    switch (fmt) {
        case T_Q8_0: lane = run_lane<T_Q8_0>; break;
        case T_Q4_K: lane = run_lane<T_Q4_K>; break;
        case T_Q5_K: lane = run_lane<T_Q5_K>; break;
        case T_Q6_K: lane = run_lane<T_Q6_K>; break;
        case T_Q2_K: lane = run_lane<T_Q2_K>; break;
        case T_IQ4_XS: lane = run_lane<T_IQ4_XS>; break;
        case T_IQ3_XXS: lane = run_lane<T_IQ3_XXS>; memcpy(cb, q38b_iq3xxs_grid, 256 * 4); break;
        case T_IQ3_S: lane = run_lane<T_IQ3_S>; memcpy(cb, q38b_iq3s_grid, 512 * 4); break;
        case T_IQ2_XXS: lane = run_lane<T_IQ2_XXS>; fill_grid<T_IQ2_XXS>(cb, q38b_iq2xxs_codes); break;
        case T_IQ2_XS: lane = run_lane<T_IQ2_XS>; fill_grid<T_IQ2_XS>(cb, q38b_iq2xs_codes); break;
        case T_IQ2_S: lane = run_lane<T_IQ2_S>; fill_grid<T_IQ2_S>(cb, q38b_iq2s_codes); break;
        case T_IQ1_S: lane = run_lane<T_IQ1_S>; fill_grid<T_IQ1_S>(cb, q38b_iq1s_codes); break;
        case T_IQ1_M: lane = run_lane<T_IQ1_M>; fill_grid<T_IQ1_M>(cb, q38b_iq1s_codes); break;
        default: return -1;
    }
    Job job{nsb, nb, slot, shift, st, actq, cb, sgn, zero, bsum, actd.data(), y};
    pthread_barrier_init(&g_bar, nullptr, 32);
    pthread_t th[32];
    Lane la[32];
    for (int l = 0; l < 32; l++) { la[l] = {&job, l}; pthread_create(&th[l], nullptr, lane, &la[l]); }
    for (int l = 0; l < 32; l++) pthread_join(th[l], nullptr);
    pthread_barrier_destroy(&g_bar);
    return 0;
}
