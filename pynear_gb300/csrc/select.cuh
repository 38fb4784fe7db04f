// select.cuh — warp-level selection over unordered 64-bit (distance, index) keys.
//
// Where many candidates were collected without order, sorting or counting them
// once is cheaper than keeping an ordered list while they arrive (topk.cuh).
#pragma once

#include "common.cuh"

namespace gn {

// Ascending bitonic sort of 32 R keys, element r * 32 + lane in v[r].
template <int R>
__device__ __forceinline__ void warp_sort(uint64_t (&v)[R]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32 * R; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 32) {
                const int rs = stride / 32;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r & rs) continue;
                    const bool up = ((r * 32) & size) == 0;  // size > stride >= 32: the lane has no say
                    const uint64_t a = v[r], b = v[r | rs];
                    const bool swap = (a > b) == up;
                    v[r] = swap ? b : a;
                    v[r | rs] = swap ? a : b;
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint64_t o = __shfl_xor_sync(0xffffffffu, v[r], stride);
                    const bool up = ((r * 32 + lane) & size) == 0;
                    const bool low = (lane & stride) == 0;
                    const bool keep_min = up == low;
                    v[r] = keep_min == (o < v[r]) ? o : v[r];
                }
            }
        }
    }
}

// The S smallest of a warp's m keys (all distinct) without order: returns a key
// such that exactly min(S, m) keys are at or below it.  The keys are lane-strided
// in registers (key i * 32 + lane in v[i], KEY_EMPTY past m).  The distance part
// of the bound is built bit by bit, from the highest bit in which the distances
// differ, out of the count of keys below each trial value; it is done as soon as
// one trial has exactly S below it (ten-odd steps for a few hundred float
// distances).  Only where keys share the S-th distance do further steps settle
// the index.  (Inserting ~400 keys into an ordered register list took about 130
// insertions of 40 instructions.)
template <int R>
__device__ __forceinline__ uint64_t warp_select(const uint64_t (&v)[R], int m, int S) {
    if (m <= S) return KEY_EMPTY - 1;
    uint32_t any = 0u, all = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (v[i] != KEY_EMPTY) {
            any |= key_dist(v[i]);
            all &= key_dist(v[i]);
        }
    any = __reduce_or_sync(0xffffffffu, any);
    all = __reduce_and_sync(0xffffffffu, all);
    uint32_t dist = all;
    int below = 0;  // keys nearer than `dist`
    if (any != all) {
        int bit = 31 - __clz((int)(any ^ all));
        dist = bit == 31 ? 0u : all & ~((2u << bit) - 1u);
#pragma unroll 1
        for (; bit >= 0; --bit) {
            const uint32_t trial = dist | (1u << bit);
            int c = 0;
#pragma unroll
            for (int i = 0; i < R; ++i) c += key_dist(v[i]) < trial;
            c = __reduce_add_sync(0xffffffffu, c);
            if (c == S) return make_key(trial - 1u, 0xffffffffu);
            if (c < S) {
                dist = trial;
                below = c;
            }
        }
    }
    const int want = S - below;  // of the keys at this distance, the lowest indices
    uint32_t idx = 0;
#pragma unroll 1
    for (int bit = 31; bit >= 0; --bit) {
        const uint32_t trial = idx | (1u << bit);
        int c = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) c += key_dist(v[i]) == dist && key_idx(v[i]) < trial;
        if (__reduce_add_sync(0xffffffffu, c) < want) idx = trial;
    }
    return make_key(dist, idx);
}

// One round of warp_best: the S best of the `kept` keys in sel and the `take` keys
// get(0) .. (at most 32 R together) into sel.
template <int R, typename Get>
__device__ __forceinline__ int warp_best_round(Get &&get, int take, int kept, int S, uint64_t *sel) {
    const int lane = threadIdx.x & 31;
    uint64_t v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int x = i * 32 + lane;
        v[i] = x < kept ? sel[x] : x - kept < take ? get(x - kept) : KEY_EMPTY;
    }
    const uint64_t thr = warp_select<R>(v, kept + take, S);
    __syncwarp();
    kept = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const bool in = v[i] <= thr && v[i] != KEY_EMPTY;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) sel[kept + __popc(b & ((1u << lane) - 1))] = v[i];
        kept += __popc(b);
    }
    __syncwarp();
    return kept;
}

// The S best of m keys get(0) .. get(m - 1) into sel[0 .. min(S, m)), any order, by
// one warp; returns their number.  S <= 256.
constexpr int SEL_R = 16;  // keys per lane held in registers at a time
template <typename Get>
__device__ __forceinline__ int warp_best_of(Get &&get, int m, int S, uint64_t *sel) {
    if (m <= 128) return warp_best_round<4>(get, m, 0, S, sel);
    int kept = 0;
    for (int i0 = 0; i0 < m;) {  // earlier rounds' best join each round's keys
        const int take = min(m - i0, SEL_R * 32 - kept);
        kept = warp_best_round<SEL_R>([&](int i) { return get(i0 + i); }, take, kept, S, sel);
        i0 += take;
    }
    return kept;
}
__device__ __forceinline__ int warp_best(const uint64_t *p, int m, int S, uint64_t *sel) {
    return warp_best_of([&](int i) { return p[i]; }, m, S, sel);
}

// ── unordered candidate buffers ───────────────────────────────────────────
// A list keeps its candidates without order in a buffer of LIST_CAP_S (k <= 64) or
// LIST_CAP_L (k <= 256) keys; one that holds more than `most` is cut to its k best.
constexpr int LIST_CAP_S = 128, LIST_CAP_L = 512;
__host__ __device__ inline int list_cap(int k) { return k <= 64 ? LIST_CAP_S : LIST_CAP_L; }
// a late cut leaves the threshold loose, an early one is paid more often (and
// appending adds up to 32 keys before the next check)
__host__ __device__ inline int list_most(int k) {
    return k > 64 ? LIST_CAP_L - 32 : 2 * k + 24 < LIST_CAP_S - 32 ? 2 * k + 24 : LIST_CAP_S - 32;
}

// Cut a buffer of m keys (k < m <= 32 R) down to its k best, in place; returns
// the k-th best key's distance bits.  (A call, not inlined: it runs a few times
// per list and would crowd the scan's registers and instruction cache.)
template <int R>
__device__ __noinline__ uint32_t list_cut(uint64_t *buf, int m, int k) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    uint64_t v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = i * 32 + lane < m ? buf[i * 32 + lane] : KEY_EMPTY;
    const uint64_t thr = warp_select<R>(v, m, k);
    __syncwarp();
    int kept = 0;
    uint32_t far = 0u;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const bool in = v[i] <= thr && v[i] != KEY_EMPTY;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) {
            buf[kept + __popc(b & ((1u << lane) - 1))] = v[i];
            far = max(far, key_dist(v[i]));
        }
        kept += __popc(b);
    }
    __syncwarp();
    return __reduce_max_sync(0xffffffffu, far);
}
__device__ __forceinline__ uint32_t list_cut_k(uint64_t *buf, int m, int k) {
    return k <= 64 ? list_cut<LIST_CAP_S / 32>(buf, m, k) : list_cut<LIST_CAP_L / 32>(buf, m, k);
}

// Add the lanes' (bits, index) keys with bits below the threshold state.y to a
// list of state.x keys, cutting it once it holds more than `most`.  ASCENDING:
// indices come in ascending order, so after a cut only smaller bits displace the
// k-th; otherwise equal bits may too, by a lower index.
template <bool ASCENDING>
__device__ __forceinline__ uint2 list_add(uint64_t *buf, uint2 state, uint32_t bits, bool in, uint32_t index, int k,
                                          int most) {
    in = in && bits < state.y;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    const int lane = threadIdx.x & 31;
    if (in) buf[state.x + __popc(m & ((1u << lane) - 1))] = make_key(bits, index);
    state.x += __popc(m);
    if ((int)state.x > most) {
        state.y = list_cut_k(buf, state.x, k) + (ASCENDING ? 0u : 1u);
        state.x = k;
    }
    return state;
}

}  // namespace gn
