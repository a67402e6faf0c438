// q38b_topk.cuh -- the k largest logits of a vector with their positions, sorted (k <= 64).
//
// Replaces topk of the reference's sampling step (src/cuda/ops.cuh:142-144, src/cuda/ops.cu:823-903,1037-1044; called on
// the output head's logits, src/runtime/engine.cpp:1680,1910): the same result -- values descending, equal values by
// ascending position -- from a different construction.  A logit becomes a 32-bit key whose unsigned order is the float
// order (NaN lowest), so that a warp's maximum is one REDUX and the tie-break a second one; no shuffle ladders.
//   stage 1: one warp per 1024 logits (32 per lane, in registers) finds its k-th largest key bit by bit -- a count of the
//            keys at or above a candidate per bit -- and emits the keys above it and the first of the keys equal to it,
//            in the order of their positions;
//   stage 2: one CTA does the same over all lists, then every survivor counts the survivors before it: its place.
// Both are chains of about 25 dependent steps of some 100 clocks (where more than k keys reach the k-th, stage 2 searches
// 31 steps more for the last position), whatever k is.  Up to TOPK_FEW elements are picked one after the other instead,
// 0.45 us an element in both stages together: stage 1 keeps each lane's largest key and looks for its next one when the
// warp has picked it, stage 2 lets every 256 candidates emit their best as a list and merges the heads of the lists.  Both
// stages, 248320 logits, one column: k = 1 10.0 us (searched: 17.7), k = 8 13.3 (17.4), k = 16 17.9 (picked: 18.7; eight
// columns 22.1 and 27.3), k = 32 20.1, k = 64 29.9.  (An earlier version that picked every k took 11.4 to 75.5 us.)
#pragma once
#include <cstdint>

namespace q38b {

constexpr int TOPK_MAX_K = 64;
constexpr int TOPK_CHUNK = 1024;
constexpr int TOPK_MAX_CHUNKS = 384;
constexpr int TOPK_STAGE1_WARPS = 2;          // 243 chunks of a 248320-word vocabulary over 148 SMs
constexpr int TOPK_MERGE_THREADS = 1024;
constexpr int TOPK_FEW = 8;                   // elements that are picked one by one, at most
constexpr int TOPK_MAX_ROUNDS = TOPK_MAX_CHUNKS * TOPK_MAX_K / TOPK_MERGE_THREADS;   // candidates per thread of stage 2

// unsigned order == float order (-0 and +0 are one key, as they compare equal); every NaN maps to 0, below -inf (0x007FFFFF)
__device__ __forceinline__ uint32_t topk_key(float f) {
    uint32_t u = __float_as_uint(f);
    if ((u & 0x7FFFFFFFu) > 0x7F800000u) return 0u;
    if (u == 0x80000000u) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

struct TopkPair { uint32_t key; int idx; };   // idx = 0x7fffffff: nothing (a list shorter than k)

// The bits of the k-th key that are known from bounds lo <= k-th key <= hi: where the two differ first, and what is above.
struct TopkStart { int bit; uint32_t t; };   // bit < 0: nothing is open, t is the key
__device__ __forceinline__ TopkStart topk_start(uint32_t lo, uint32_t hi) {
    const int bit = 31 - __clz((int)(lo ^ hi));
    return TopkStart{bit, bit < 0 ? hi : hi & ~((2u << bit) - 1u)};
}

// grid (chunks, columns).  lists: [column][chunk][k] pairs by ascending position (up to TOPK_FEW: best first), then empty ones.
template <bool FEW>
static __global__ void __launch_bounds__(TOPK_STAGE1_WARPS * 32) topk_lists_kernel(const float* __restrict__ x, long long x_ld, int n, int k,
                                                                             TopkPair* __restrict__ lists, int n_chunks) {
    const int lane = threadIdx.x & 31;
    const int chunk = blockIdx.x * TOPK_STAGE1_WARPS + (threadIdx.x >> 5);
    if (chunk >= n_chunks) return;
    const float* xc = x + (size_t)blockIdx.y * x_ld;
    const int base = chunk * TOPK_CHUNK, here = min(TOPK_CHUNK, n - base);
    uint32_t key[32];
#pragma unroll
    for (int j = 0; j < 32; j++) {
        const int i = 32 * j + lane;
        key[j] = i < here ? topk_key(xc[base + i]) : 0u;
    }
    if constexpr (FEW) {
        uint32_t live = 0u;                     // bit j: element j exists and has not been picked (its key is 0 afterwards)
#pragma unroll
        for (int j = 0; j < 32; j++) live |= (32 * j + lane < here ? 1u : 0u) << j;
        uint32_t best = 0u;
        int slot = -1;                          // this lane's largest key and its first place; -1: nothing left
        auto scan = [&]() {
            uint32_t m4[4] = {0u, 0u, 0u, 0u}, at = 0u;
#pragma unroll
            for (int j = 0; j < 32; j++) m4[j & 3] = max(m4[j & 3], key[j]);
            best = max(max(m4[0], m4[1]), max(m4[2], m4[3]));
#pragma unroll
            for (int j = 0; j < 32; j++) at |= (key[j] == best ? 1u : 0u) << j;
            slot = __ffs((int)(at & live)) - 1;
        };
        scan();
        TopkPair mine{0u, 0x7fffffff};
        for (int r = 0; r < k; r++) {
            const uint32_t w = __reduce_max_sync(0xffffffffu, best);
            const int p = slot >= 0 && best == w ? base + 32 * slot + lane : 0x7fffffff;
            const int first = (int)__reduce_min_sync(0xffffffffu, (unsigned)p);
            if (lane == r) mine = TopkPair{w, first};
            if (p == first && p != 0x7fffffff) {
                live &= ~(1u << slot);
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (j == slot) key[j] = 0u;
                scan();
            }
        }
        if (lane < k) lists[((size_t)blockIdx.y * n_chunks + chunk) * k + lane] = mine;
        return;
    }
    // the largest t that at least k keys reach (0 when fewer are above 0: NaN logits fill up); keys past the end are 0
    // (the lanes' largest keys are 32 keys: at least k <= 32 reach the smallest of them)
    uint32_t top = 0u;
#pragma unroll
    for (int j = 0; j < 32; j++) top = max(top, key[j]);
    const TopkStart start = topk_start(k <= 32 ? __reduce_min_sync(0xffffffffu, top) : 0u, __reduce_max_sync(0xffffffffu, top));
    uint32_t t = start.t;
    for (int bit = start.bit; bit >= 0; bit--) {
        const uint32_t cand = t | (1u << bit);
        int c4[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < 32; j++) c4[j & 3] += key[j] >= cand;
        const int c = (int)__reduce_add_sync(0xffffffffu, (unsigned)((c4[0] + c4[1]) + (c4[2] + c4[3])));
        if (c >= k) t = cand;
        if (c == k) break;
    }
    int above = 0;
#pragma unroll
    for (int j = 0; j < 32; j++) above += key[j] > t;
    int ties = k - (int)__reduce_add_sync(0xffffffffu, (unsigned)above);   // how many keys equal to t are taken: the earliest
    TopkPair* out = lists + ((size_t)blockIdx.y * n_chunks + chunk) * k;
    const uint32_t before = (1u << lane) - 1u;
    int at = 0;
#pragma unroll
    for (int j = 0; j < 32; j++) {
        const int i = 32 * j + lane;
        const bool equal = key[j] == t && i < here;
        const uint32_t eq = __ballot_sync(0xffffffffu, equal);
        const bool take = key[j] > t || (equal && __popc(eq & before) < ties);
        ties -= min(ties, __popc(eq));
        const uint32_t tk = __ballot_sync(0xffffffffu, take);
        if (take) out[at + __popc(tk & before)] = TopkPair{key[j], base + i};
        at += __popc(tk);
    }
    for (int r = at + lane; r < k; r += 32) out[r] = TopkPair{0u, 0x7fffffff};
}

// Stage 2 for k <= TOPK_FEW: grid (columns), a warp per 256 candidates.
constexpr int TOPK_FEW_ROUNDS = 8;
static_assert(TOPK_MAX_CHUNKS * TOPK_FEW <= 32 * 32 * TOPK_FEW_ROUNDS && TOPK_FEW <= 32, "a list per lane, a result per lane");
static __global__ void __launch_bounds__(1024) topk_merge_few_kernel(const TopkPair* __restrict__ lists, int n_chunks, int k, const float* __restrict__ x,
                                                                     long long x_ld, int index_offset, float* __restrict__ vals, int* __restrict__ idx,
                                                                     long long out_ld) {
    __shared__ TopkPair heads[32 * TOPK_FEW];
    const TopkPair* src = lists + (size_t)blockIdx.x * n_chunks * k;
    const int total = n_chunks * k, warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31, n_warps = (int)blockDim.x >> 5;
    const TopkPair none{0u, 0x7fffffff};
    uint32_t key[TOPK_FEW_ROUNDS];
    int pos[TOPK_FEW_ROUNDS];
#pragma unroll
    for (int r = 0; r < TOPK_FEW_ROUNDS; r++) {
        const int i = 32 * (TOPK_FEW_ROUNDS * warp + r) + lane;
        const TopkPair p = i < total ? src[i] : none;
        key[r] = p.key;
        pos[r] = p.idx;
    }
    TopkPair mine = none;
    for (int t = 0; t < k; t++) {
        uint32_t best = 0u;
        int at = 0x7fffffff;
#pragma unroll
        for (int r = 0; r < TOPK_FEW_ROUNDS; r++) best = max(best, key[r]);
#pragma unroll
        for (int r = 0; r < TOPK_FEW_ROUNDS; r++) at = min(at, key[r] == best ? pos[r] : 0x7fffffff);
        const uint32_t w = __reduce_max_sync(0xffffffffu, best);
        const int first = (int)__reduce_min_sync(0xffffffffu, (unsigned)(best == w ? at : 0x7fffffff));
        if (lane == t) mine = TopkPair{w, first};
#pragma unroll
        for (int r = 0; r < TOPK_FEW_ROUNDS; r++)
            if (pos[r] == first) { key[r] = 0u; pos[r] = 0x7fffffff; }
    }
    if (lane < k) heads[warp * k + lane] = mine;
    __syncthreads();
    if (warp > 0) return;
    int taken = 0;
    TopkPair head = lane < n_warps ? heads[lane * k] : none;
    mine = none;
    for (int t = 0; t < k; t++) {
        const uint32_t w = __reduce_max_sync(0xffffffffu, head.key);
        const int first = (int)__reduce_min_sync(0xffffffffu, (unsigned)(head.key == w ? head.idx : 0x7fffffff));
        if (lane == t) mine = TopkPair{w, first};
        if (head.idx == first && first != 0x7fffffff) head = ++taken < k ? heads[lane * k + taken] : none;
    }
    if (lane >= k) return;
    const bool empty = mine.idx == 0x7fffffff;
    vals[(size_t)blockIdx.x * out_ld + lane] = empty ? __uint_as_float(0x7FC00000u) : x[(size_t)blockIdx.x * x_ld + mine.idx];
    idx[(size_t)blockIdx.x * out_ld + lane] = empty ? -1 : mine.idx + index_offset;
}

// Sum over the CTA of one count per thread; `slots`: [2][32] ints, used alternately so that one barrier per sum is enough.
__device__ __forceinline__ int topk_cta_sum(int c, int* slots, int& phase) {
    c = (int)__reduce_add_sync(0xffffffffu, (unsigned)c);
    int* s = slots + 32 * phase;
    phase ^= 1;
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    return (int)__reduce_add_sync(0xffffffffu, (unsigned)s[threadIdx.x & 31]);
}

// grid (columns), one CTA.  vals / idx: [column][ld] floats and ints.  ROUNDS: candidates per thread.
template <int ROUNDS>
static __global__ void __launch_bounds__(TOPK_MERGE_THREADS) topk_merge_kernel(const TopkPair* __restrict__ lists, int n_chunks, int k,
                                                                               const float* __restrict__ x, long long x_ld, int index_offset,
                                                                               float* __restrict__ vals, int* __restrict__ idx, long long out_ld) {
    static_assert(TOPK_MERGE_THREADS == 1024, "one count per warp fills a warp");
    __shared__ int slots[64];
    __shared__ int n_best;
    __shared__ TopkPair best[TOPK_MAX_K];
    const TopkPair* src = lists + (size_t)blockIdx.x * n_chunks * k;
    const int total = n_chunks * k;
    uint32_t key[ROUNDS];
    int pos[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int i = r * TOPK_MERGE_THREADS + (int)threadIdx.x;
        const TopkPair p = i < total ? src[i] : TopkPair{0u, 0x7fffffff};
        key[r] = p.key;
        pos[r] = p.idx;
    }
    if (threadIdx.x == 0) n_best = 0;
    // the same bounds from the largest key of each of the 32 warps
    uint32_t top = 0u;
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) top = max(top, key[r]);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = (int)top;
    __syncthreads();
    top = (uint32_t)slots[threadIdx.x & 31];
    const TopkStart start = topk_start(k <= 32 ? __reduce_min_sync(0xffffffffu, top) : 0u, __reduce_max_sync(0xffffffffu, top));
    int phase = 1, c_t = -1;
    uint32_t t = start.t;
    for (int bit = start.bit; bit >= 0 && c_t != k; bit--) {
        const uint32_t cand = t | (1u << bit);
        int c = 0;
#pragma unroll
        for (int r = 0; r < ROUNDS; r++) c += key[r] >= cand;
        c = topk_cta_sum(c, slots, phase);
        if (c >= k) { t = cand; c_t = c; }
    }
    // among the keys equal to t the earliest positions: the smallest `last` that leaves k elements (none missing: all of them)
    int last = 0x7ffffffe;
    if (c_t != k) {
        last = 0;
        for (int bit = 30; bit >= 0; bit--) {   // the smallest last with count(last) >= k, as the largest value below it plus one
            const int cand = last | (1 << bit);
            int c = 0;
#pragma unroll
            for (int r = 0; r < ROUNDS; r++) c += key[r] > t || (key[r] == t && pos[r] < cand);
            c = topk_cta_sum(c, slots, phase);
            if (c < k) last = cand;
        }
        last = min(last, 0x7ffffffe);           // positions below or at `last`; empty list entries (0x7fffffff) never
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; r++)
        if (key[r] > t || (key[r] == t && pos[r] <= last)) {
            const int s = atomicAdd(&n_best, 1);
            if (s < k) best[s] = TopkPair{key[r], pos[r]};
        }
    __syncthreads();
    const int m = min(n_best, k), i = (int)threadIdx.x;
    if (i >= k) return;
    float* ov = vals + (size_t)blockIdx.x * out_ld;
    int* oi = idx + (size_t)blockIdx.x * out_ld;
    if (i >= m) {
        ov[i] = __uint_as_float(0x7FC00000u);
        oi[i] = -1;
        return;
    }
    const TopkPair me = best[i];
    int place = 0;
    for (int j = 0; j < m; j++) place += best[j].key > me.key || (best[j].key == me.key && best[j].idx < me.idx);
    ov[place] = x[(size_t)blockIdx.x * x_ld + me.idx];   // the logit itself (the key does not keep -0 or NaN payloads)
    oi[place] = me.idx + index_offset;
}

}  // namespace q38b
