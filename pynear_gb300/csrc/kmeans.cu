// kmeans.cu — float and binary k-means on the device.
//
// Float (replaces kmeans_l2, pynear/include/KMeans.hpp:25-126):
//   seeding   k-means++ exactly as the reference: mt19937(seed) draws on the
//             host (taken up front: they do not depend on the data), squared
//             dist_l2_f_avx2 distances computed on the device in the
//             reference's arithmetic order, the weighted pick on the device
//             from double running sums, with the reference's serial double
//             sums deciding where the two orders could disagree (so the seeds
//             are the reference's);
//   assign    argmin_c (|c|^2 - 2 x.c) from an FP32 tile GEMM with a fused
//             argmin epilogue (first minimum wins, like the reference);
//   update    per-cluster sums in FP64 (atomic adds), divided once and rounded
//             to float; empty clusters re-seeded with pick_point(rng) in
//             cluster order, as the reference does.
// Binary (replaces IVFFlatBinaryIndex::_build, pynear/include/BinaryIVF.hpp:
// 127-227): integer arithmetic throughout, so the device build reproduces the
// reference's centroids and labels exactly: the same mt19937 stream (pick, then
// wsel over [0,total)), exact int64 sums and prefix search, first-minimum
// Hamming assignment, majority vote count > n_c/2, empty clusters re-seeded.
#include <algorithm>
#include <cstring>
#include <random>
#include <vector>

#include "distance.cuh"
#include "gemm_topk.cuh"
#include "index.cuh"
#include "kmeans.cuh"

namespace gn {

// ── block reductions of the seeding kernels (256 threads) ─────────────────
constexpr int KPP_NT = 256;
constexpr int KPP_ROWS = KPP_NT / 2;  // rows a block of the float seeding takes at a time
constexpr int KPP_SPAN = 4;           // chunk sums per thread of the pick: at most KPP_NT * KPP_SPAN chunks

// Exclusive block-wide scan; *total = the sum of all threads' v.  Threads from
// `active` on hold zero: their warps add nothing (FP64 runs at two lanes per
// clock and SM, so additions of zeros would cost as much as the others).
template <typename T>
__device__ __forceinline__ T kpp_block_scan(T v, T *total, int active = KPP_NT) {
    __shared__ T wsum[KPP_NT / 32 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = v;
    if (warp * 32 < active) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
    }
    __syncthreads();  // wsum of an earlier call is no longer read
    if (lane == 31) wsum[warp + 1] = inc;
    __syncthreads();
    if (warp == 0) {
        T w = lane < KPP_NT / 32 ? wsum[lane + 1] : T(0);
#pragma unroll
        for (int o = 1; o < KPP_NT / 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < KPP_NT / 32) wsum[lane + 1] = w;
        if (lane == 0) wsum[0] = T(0);
    }
    __syncthreads();
    *total = wsum[KPP_NT / 32];
    return warp * 32 < active ? wsum[warp] + (inc - v) : wsum[KPP_NT / 32];
}

// True in every thread of the launch's last block to arrive (whose view then
// holds what the others wrote before they arrived); resets the counter.
__device__ __forceinline__ bool kpp_last_block(unsigned *done) {
    __shared__ unsigned s_arrival;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_arrival = atomicAdd(done, 1u);
    __syncthreads();
    const bool last = s_arrival == gridDim.x - 1;
    if (last) {
        __threadfence();
        if (threadIdx.x == 0) *done = 0;
    }
    return last;
}

// ── float seeding ─────────────────────────────────────────────────────────
// The reference's serial draw (KMeans.hpp:45-70), by one thread: the first row whose
// running sum in double reaches u times the sum of all.  A chain of additions as long as
// the rows; the values are loaded 16 ahead, or each would wait for its load too (344,491
// rows: 46 ms, 25 so).
__device__ __noinline__ int64_t kpp_serial(const float *min_sq, int64_t n, float u) {
    constexpr int AHEAD = 16;
    auto load = [&](int64_t i0, float (&v)[AHEAD]) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) v[i] = i0 + i < n ? __ldcg(min_sq + i0 + i) : 0.f;
    };
    float v[AHEAD];
    double total = 0.0, sum = 0.0;
    for (int64_t i0 = 0; i0 < n; i0 += AHEAD) {
        load(i0, v);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) total += (double)v[i];
    }
    const double target = (double)u * total;
    for (int64_t i0 = 0; i0 < n; i0 += AHEAD) {
        load(i0, v);
        double at[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) at[i] = sum = sum + (double)v[i];
        if (sum < target) continue;  // (the values are not negative: nor are the sums before)
        for (int i = 0; i < AHEAD && i0 + i < n; ++i)
            if (at[i] >= target) return i0 + i;
    }
    return n - 1;
}

// One launch per k-means++ draw, for rows past the SMs' shared memory (see
// kpp_seed_kernel for the others): every block lowers its chunk's min_sq by the
// distances to the newest centroid (row ci - 1 of C) and sums the chunk in
// double; the last block to finish draws centroid ci and copies its row.
//
// Two threads per row, each with four of the reference's eight accumulators:
// a warp's 16-byte loads cover whole 32-byte sectors (a thread per row read
// 16 bytes of 32 different lines at a time), and the two halves meet in the
// fold that the reference's order has anyway (lane j + 4 onto lane j).
//
// The draw is the reference's rule (KMeans.hpp:45-70): r = u * sum(min_sq), the
// first point whose running sum reaches r (n - 1 if none).  The reference sums
// in double in point order; here the sums are the chunk sums, scanned, then
// the chosen chunk's elements.  Both orders' running sums lie within
// 2 (n - 1) 2^-53 total of the exact ones, so when r is farther than twice that
// from the chosen point's running sums on both sides, the serial order chooses
// the same point; if not, thread 0 repeats the reference's serial loop (rare).
// What bounds it is the chain of dependent FP64 additions (the unit's latency,
// not its rate), so every sum is a scan over lanes: 100k x 64, 255 draws:
// 12.2 ms as three launches with serial sums over the warps' totals, 3.8 ms
// as this one.
__global__ void __launch_bounds__(KPP_NT) kpp_kernel(const float *__restrict__ X, int64_t n, int d, int dp,
                                                     float *__restrict__ C, int64_t ci, float u,
                                                     float *__restrict__ min_sq, int64_t chunk, int P,
                                                     double *__restrict__ part, unsigned *__restrict__ done) {
    const int t = threadIdx.x;
    const int64_t b0 = (int64_t)blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    __shared__ float s_m[KPP_ROWS];
    {
        const int half = t & 1;
        const int nb = d >> 3, rem = d & 7, dp4 = dp >> 2;
        const float4 *c4 = reinterpret_cast<const float4 *>(C) + (ci - 1) * dp4;
        const float4 *x4 = reinterpret_cast<const float4 *>(X);
        double s = 0.0;  // warp 0: this lane's share of the chunk's sum
        for (int64_t i0 = b0; i0 < b1; i0 += KPP_ROWS) {
            const int64_t i = i0 + (t >> 1);
            const bool in = i < b1;
            const float4 *xr = x4 + (in ? i : b0) * dp4 + half;
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll 8
            for (int c = 0; c < nb; ++c) {
                const float4 x = xr[2 * c], q = c4[2 * c + half];
                const float t0 = __fsub_rn(q.x, x.x), t1 = __fsub_rn(q.y, x.y);
                const float t2 = __fsub_rn(q.z, x.z), t3 = __fsub_rn(q.w, x.w);
                a0 = __fmaf_rn(t0, t0, a0);
                a1 = __fmaf_rn(t1, t1, a1);
                a2 = __fmaf_rn(t2, t2, a2);
                a3 = __fmaf_rn(t3, t3, a3);
            }
            float s0 = __fadd_rn(a0, __shfl_xor_sync(0xffffffffu, a0, 1));
            float s1 = __fadd_rn(a1, __shfl_xor_sync(0xffffffffu, a1, 1));
            float s2 = __fadd_rn(a2, __shfl_xor_sync(0xffffffffu, a2, 1));
            float s3 = __fadd_rn(a3, __shfl_xor_sync(0xffffffffu, a3, 1));
            // the 4-wide step and the masked remainder (rows are zero padded past d)
            for (int w = 0; 4 * w < rem; ++w) {
                const float4 x = x4[(in ? i : b0) * dp4 + 2 * nb + w], q = c4[2 * nb + w];
                const float t0 = __fsub_rn(q.x, x.x), t1 = __fsub_rn(q.y, x.y);
                const float t2 = __fsub_rn(q.z, x.z), t3 = __fsub_rn(q.w, x.w);
                s0 = __fmaf_rn(t0, t0, s0);
                s1 = __fmaf_rn(t1, t1, s1);
                s2 = __fmaf_rn(t2, t2, s2);
                s3 = __fmaf_rn(t3, t3, s3);
            }
            if (half == 0) {
                float m = 0.f;
                if (in) {
                    const float r = __fsqrt_rn(__fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2, s3)));
                    const float v = __fmul_rn(r, r);
                    m = ci == 1 ? 3.402823466e+38f : min_sq[i];
                    if (v < m || ci == 1) {
                        m = v < m ? v : m;
                        min_sq[i] = m;
                    }
                }
                s_m[t >> 1] = m;
            }
            // the step's 128 values in double by one warp (see kpp_block_scan on FP64's rate)
            __syncthreads();
            if (t < 32) {
                s += ((double)s_m[t] + (double)s_m[t + 32]) + ((double)s_m[t + 64] + (double)s_m[t + 96]);
                __syncwarp();
            }
            if (i0 + KPP_ROWS < b1) __syncthreads();
        }
        if (t < 32) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (t == 0) part[blockIdx.x] = s;
        }
    }
    if (!kpp_last_block(done)) return;

    __shared__ int s_b, s_amb, s_found;
    __shared__ double s_base;
    __shared__ unsigned long long s_chosen;
    if (t == 0) {
        s_b = P;
        s_amb = 0;
        s_found = 0;
        s_base = 0.0;
        s_chosen = (unsigned long long)(n - 1);
    }
    // the chunk that holds the point: every thread has KPP_SPAN neighbouring chunk sums
    double ps[KPP_SPAN];
#pragma unroll
    for (int i = 0; i < KPP_SPAN; ++i) {
        const int p = t * KPP_SPAN + i;
        ps[i] = p < P ? __ldcg(part + p) : 0.0;
    }
    const int pick_threads = (P + KPP_SPAN - 1) / KPP_SPAN;
    double own = 0.0;
    if ((t & ~31) < pick_threads) own = (ps[0] + ps[1]) + (ps[2] + ps[3]);
    double total;
    const double pre = kpp_block_scan(own, &total, pick_threads);
    const double r = (double)u * total;
    const double band = 4.0 * (double)n * 1.1102230246251565e-16 * total;  // 2 x 2 (n - 1) 2^-53 total, rounded up
    int mine = P;
    double mbase = 0.0;
    if ((t & ~31) < pick_threads) {
        double cum = pre;
#pragma unroll
        for (int i = 0; i < KPP_SPAN; ++i) {
            const double nx = cum + ps[i];
            if (mine == P && nx >= r && t * KPP_SPAN + i < P) {
                mine = t * KPP_SPAN + i;
                mbase = cum;
            }
            cum = nx;
        }
    }
    if (mine < P) atomicMin(&s_b, mine);
    __syncthreads();
    const int b = s_b;
    if (b < P && mine == b) s_base = mbase;
    __syncthreads();
    if (b < P) {
        // running sums inside chunk b: each thread takes a contiguous piece
        const int64_t c0 = (int64_t)b * chunk, c1 = min(n, c0 + chunk);
        const int64_t per = (c1 - c0 + KPP_NT - 1) / KPP_NT;
        const int64_t e0 = min(c1, c0 + t * per), e1 = min(c1, e0 + per);
        const int chunk_threads = (int)((c1 - c0 + per - 1) / per);
        double ls = 0.0;
        for (int64_t i = e0; i < e1; ++i) ls += (double)__ldcg(min_sq + i);
        double lt;
        double cum = s_base + kpp_block_scan(ls, &lt, chunk_threads);  // running sum before this thread's piece
        int64_t found = -1;
        double before = 0.0, at = 0.0;
        for (int64_t i = e0; i < e1; ++i) {
            const double nx = per == 1 ? cum + ls : cum + (double)__ldcg(min_sq + i);
            if (nx >= r) {
                found = i;
                before = cum;
                at = nx;
                break;
            }
            cum = nx;
        }
        // the first piece holding the point: pieces are ordered, so the lowest index wins
        if (found >= 0) {
            atomicMin(&s_chosen, (unsigned long long)found);
            s_found = 1;
        }
        __syncthreads();
        if (found >= 0 && (unsigned long long)found == s_chosen && !(at - r > band && r - before > band)) s_amb = 1;
        // the chunk's elements summed in this order fell short of r: the serial rule decides
        if (t == 0 && !s_found) s_amb = 1;
    } else if (t == 0) {
        s_amb = 1;  // r beyond every partial sum: the serial rule decides
    }
    __syncthreads();
    if (s_amb && t == 0) s_chosen = (unsigned long long)kpp_serial(min_sq, n, u);
    __syncthreads();
    const int64_t ch = (int64_t)s_chosen;
    for (int j = t; j < dp; j += KPP_NT) C[ci * dp + j] = X[ch * dp + j];
}

// ── seeding in one launch ─────────────────────────────────────────────────
// All the draws of a k-means++ whose rows fit the SMs' shared memory: one
// cooperative launch, a block per SM, which keeps its rows and their distances
// there, so that a draw reads nothing but the newest centroid's row.  Between the
// blocks two words travel per draw: every block's sum, which all of them read to
// find the block that holds the point, and that block's row number.  Each word
// carries its draw's tag and is polled directly (no counter, no fence: nothing
// else is handed over), in a slot per parity: a block writes draw e + 2's sum only
// after every block has written e + 1's, hence read e's.
// What bounds a draw is the chain of these two round trips and the scans between
// them, so the sums are 64-bit integers (an FP64 addition's latency is about 140
// clocks here) of 16 or 32 rows each, left by the warps that made the distances.
// Measured: 15 us a draw for 100k x 64 rows as one launch each (9.4 us for 200k x 32
// bytes), 5.0 us here (3.9 us).
constexpr int SEED_NT = 1024;
constexpr int SEED_SPAN = 8;                   // block sums per lane: at most 32 * SEED_SPAN blocks
constexpr unsigned SEED_SPINS = 1u << 22;      // polls before a wait gives up (seconds)
constexpr size_t SEED_SMEM_MAX = 222 * 1024;   // dynamic shared memory of a block
constexpr int SEED_TAG = 40;                   // row words: draw << SEED_TAG | row
constexpr unsigned long long SEED_AGAIN = 1ull << 39;  // row word: the serial rule decides

__device__ __forceinline__ unsigned long long seed_load(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void seed_store(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Poll the row word of draw ci; false (and *err set) when the limit runs out.
__device__ __forceinline__ bool seed_wait(const unsigned long long *p, int ci, unsigned long long *word, int *err,
                                          unsigned limit = SEED_SPINS) {
    for (unsigned i = 0; i < limit; ++i) {
        *word = seed_load(p);
        if (*word >> SEED_TAG == (unsigned)ci) return true;
    }
    *reinterpret_cast<volatile int *>(err) = 1;
    return false;
}
// All G blocks' words (value << 2 | ci & 3) of draw ci, by one warp: polled together
// (five loads of a warp in flight, where one word after another took a round trip
// each), then handed over through shared memory: lane l gets values l * span .. in v.
__device__ __forceinline__ bool seed_gather(const unsigned long long *words, int G, int ci,
                                            unsigned long long *s_words, unsigned long long (&v)[SEED_SPAN],
                                            int *err) {
    const int lane = threadIdx.x & 31, span = (G + 31) / 32;
    const unsigned long long tag = ci & 3;
    bool ok = false;
#pragma unroll
    for (int i = 0; i < SEED_SPAN; ++i) v[i] = ~tag;  // not yet there
    // all blocks polling the same ten lines delay the words' own way there: 8.6 us a
    // draw without this pause, 5.0 with it (100 to 600 ns made no difference)
    __nanosleep(300);
    for (unsigned tries = 0; !ok && tries < SEED_SPINS; ++tries) {
#pragma unroll
        for (int i = 0; i < SEED_SPAN; ++i)
            if (i < span && i * 32 + lane < G && (v[i] & 3) != tag) v[i] = seed_load(words + i * 32 + lane);
        ok = true;
#pragma unroll
        for (int i = 0; i < SEED_SPAN; ++i)
            if (i < span && i * 32 + lane < G) ok = ok && (v[i] & 3) == tag;
        ok = __all_sync(0xffffffffu, ok);
    }
    if (!ok) *reinterpret_cast<volatile int *>(err) = 1;
#pragma unroll
    for (int i = 0; i < SEED_SPAN; ++i)
        if (i < span && i * 32 + lane < G) s_words[i * 32 + lane] = v[i] >> 2;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < SEED_SPAN; ++i) v[i] = i < span && lane * span + i < G ? s_words[lane * span + i] : 0ull;
    __syncwarp();
    return ok;
}
// Inclusive scan over a warp.
__device__ __forceinline__ unsigned long long seed_scan(unsigned long long v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}
// One draw, by one warp of every block: s_group holds the sums of the block's rows,
// GROUP at a time, value(i) is row i's.  aim(total, &target, &band, &word) says what is
// looked for, the first row whose running sum reaches target, and how far from both
// running sums the target has to be (or returns false, with the row word of a draw
// that needs no search).  Returns the row word, 0 if a wait gave up.
template <int GROUP, typename Value, typename Aim>
__device__ __forceinline__ unsigned long long seed_draw(unsigned long long *sums, unsigned long long *row_word, int ci,
                                                        const unsigned long long *s_group, int rows, int64_t b0,
                                                        unsigned long long *s_words, Value &&value, Aim &&aim,
                                                        int *err) {
    const int lane = threadIdx.x & 31, G = gridDim.x;
    const int groups = (rows + GROUP - 1) / GROUP, per = (groups + 31) / 32;
    const int g0 = min(groups, lane * per), g1 = min(groups, g0 + per);
    unsigned long long own = 0;
    for (int g = g0; g < g1; ++g) own += s_group[g];
    const unsigned long long end = seed_scan(own, lane);  // sum of the block's rows up to this lane's last
    if (lane == 31) seed_store(sums + blockIdx.x, end << 2 | (unsigned)(ci & 3));
    unsigned long long ps[SEED_SPAN], mine = 0;
    bool ok = seed_gather(sums, G, ci, s_words, ps, err);
#pragma unroll
    for (int i = 0; i < SEED_SPAN; ++i) mine += ps[i];
    const unsigned long long incl = seed_scan(mine, lane), total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long target, band, w = 0;
    if (aim(total, target, band, w)) {
        const int span = (G + 31) / 32;
        unsigned long long cum = incl - mine, base = 0;
        int b = G;  // the block that holds the point
#pragma unroll
        for (int i = 0; i < SEED_SPAN; ++i) {
            if (i < span && b == G && cum + ps[i] >= target && lane * span + i < G) {
                b = lane * span + i;
                base = cum;
            }
            cum += ps[i];
        }
        const unsigned has = __ballot_sync(0xffffffffu, b < G);
        const int src = has ? __ffs(has) - 1 : 0;
        b = __shfl_sync(0xffffffffu, b, src);
        base = __shfl_sync(0xffffffffu, base, src);
        if ((int)blockIdx.x == (b < G ? b : 0)) {
            // the lane whose groups reach the target, its group, then the row
            unsigned long long row = SEED_AGAIN;
            const unsigned runs = __ballot_sync(0xffffffffu, base + end >= target);
            if (b < G && runs) {
                const int l = __ffs(runs) - 1;
                unsigned long long before = base + __shfl_sync(0xffffffffu, end - own, l);
                int g = l * per;
                while (g + 1 < groups && before + s_group[g] < target) before += s_group[g++];
                const int i = g * GROUP + lane;
                const bool real = lane < GROUP && i < rows;
                const unsigned long long v = real ? value(i) : 0ull, at = before + seed_scan(v, lane);
                const unsigned hit = __ballot_sync(0xffffffffu, real && at >= target);
                const int f = hit ? __ffs(hit) - 1 : 0;
                const unsigned long long at_f = __shfl_sync(0xffffffffu, at, f),
                                         before_f = __shfl_sync(0xffffffffu, at - v, f);
                if (hit && at_f - target >= band && target - before_f > band)
                    row = (unsigned long long)(b0 + g * GROUP + f);
            }
            w = (unsigned long long)ci << SEED_TAG | row;
            if (lane == 0) seed_store(row_word, w);
        } else if (lane == 0) {
            ok = ok && seed_wait(row_word, ci, &w, err);
        }
    }
    return __all_sync(0xffffffffu, ok) ? w : 0ull;
}

// A distance as a multiple of 2^e, rounded down.
__device__ __forceinline__ unsigned long long seed_fixed(float m, int e) {
    const unsigned bits = __float_as_uint(m), x = bits >> 23;
    const unsigned long long mant = (bits & 0x7fffffu) | (x ? 0x800000u : 0u);
    const int shift = (x ? (int)x - 150 : -149) - e;
    return shift >= 0 ? mant << min(shift, 63) : mant >> min(-shift, 63);
}

// The float draws: kpp_kernel's arithmetic and rule.  The sums are exact multiples of
// 2^e, e chosen before each draw so that they stay below 2^62 (from the largest first
// distance, then from the draw before: distances only fall), so they are n 2^e at most
// below the exact ones; the target is u * total to one such step.  The reference's
// double sums lie within 2 n 2^-53 total of the exact ones, and where these bounds
// leave a doubt the serial rule decides (rare): the blocks write their distances out to
// min_sq and arrive at *done, and thread 0 of block 0 repeats the reference's loop.
// u: the draws' uniforms; words, zeroed: [2][grid] sums, [2] rows, [2] rows of the
// serial rule, [grid] largest first distances.
__global__ void __launch_bounds__(SEED_NT, 1) kpp_seed_kernel(const float *__restrict__ X, int64_t n, int d, int dp,
                                                              float *C, int k, const float *__restrict__ u,
                                                              float *min_sq, int chunk, unsigned long long *words,
                                                              unsigned *done, int *err) {
    extern __shared__ __align__(16) float seed_smem[];
    __shared__ unsigned long long s_word, s_words[32 * SEED_SPAN];
    __shared__ int s_e;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, G = gridDim.x;
    const int64_t b0 = min(n, (int64_t)blockIdx.x * chunk);
    const int rows = (int)(min(n, b0 + chunk) - b0);
    const int stride = dp + 8;  // 32 bytes past a multiple of 64: four rows' 32 bytes in different banks
    float *const s_c = seed_smem, *const s_m = s_c + dp;
    unsigned long long *const s_group = reinterpret_cast<unsigned long long *>(s_m + ((chunk + 15) & ~15));
    float *const s_x = reinterpret_cast<float *>(s_group + (chunk + 31) / 32 * 2);
    const int dp4 = dp >> 2;
    for (int i = t; i < rows * dp4; i += SEED_NT)
        *reinterpret_cast<float4 *>(s_x + (i / dp4) * stride + (i % dp4) * 4) =
            __ldg(reinterpret_cast<const float4 *>(X + b0 * dp) + i);
    for (int i = t; i < rows; i += SEED_NT) s_m[i] = 3.402823466e+38f;
    for (int j = t; j < dp; j += SEED_NT) s_c[j] = C[j];
    __syncthreads();
    const int half = t & 1, nb = d >> 3, rem = d & 7;
    const float4 *c4 = reinterpret_cast<const float4 *>(s_c);
    int e = 0;
    unsigned again = 0;
    // the sum of the 16 distances of a warp's even lanes (0 on the odd ones): three
    // 21-bit parts, so that 32 lanes' sums fit a word
    const auto group_sum = [&](int g, float m) {
        const unsigned long long f = seed_fixed(m, e);
        const unsigned a = __reduce_add_sync(0xffffffffu, (unsigned)(f & 0x1fffffu));
        const unsigned b = __reduce_add_sync(0xffffffffu, (unsigned)(f >> 21 & 0x1fffffu));
        const unsigned c = __reduce_add_sync(0xffffffffu, (unsigned)(f >> 42));
        if (lane == 0) s_group[g] = ((unsigned long long)c << 42) + ((unsigned long long)b << 21) + a;
    };
    for (int ci = 1; ci < k; ++ci) {
        for (int g = warp; g * 16 < rows; g += SEED_NT / 32) {  // 16 rows a warp, two lanes a row
            const int i = g * 16 + (lane >> 1);
            const bool in = i < rows;
            const float4 *x4 = reinterpret_cast<const float4 *>(s_x + (in ? i : 0) * stride);
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll 4
            for (int c = 0; c < nb; ++c) {
                const float4 x = x4[2 * c + half], q = c4[2 * c + half];
                const float t0 = __fsub_rn(q.x, x.x), t1 = __fsub_rn(q.y, x.y);
                const float t2 = __fsub_rn(q.z, x.z), t3 = __fsub_rn(q.w, x.w);
                a0 = __fmaf_rn(t0, t0, a0);
                a1 = __fmaf_rn(t1, t1, a1);
                a2 = __fmaf_rn(t2, t2, a2);
                a3 = __fmaf_rn(t3, t3, a3);
            }
            float s0 = __fadd_rn(a0, __shfl_xor_sync(0xffffffffu, a0, 1));
            float s1 = __fadd_rn(a1, __shfl_xor_sync(0xffffffffu, a1, 1));
            float s2 = __fadd_rn(a2, __shfl_xor_sync(0xffffffffu, a2, 1));
            float s3 = __fadd_rn(a3, __shfl_xor_sync(0xffffffffu, a3, 1));
            for (int w = 0; 4 * w < rem; ++w) {
                const float4 x = x4[2 * nb + w], q = c4[2 * nb + w];
                const float t0 = __fsub_rn(q.x, x.x), t1 = __fsub_rn(q.y, x.y);
                const float t2 = __fsub_rn(q.z, x.z), t3 = __fsub_rn(q.w, x.w);
                s0 = __fmaf_rn(t0, t0, s0);
                s1 = __fmaf_rn(t1, t1, s1);
                s2 = __fmaf_rn(t2, t2, s2);
                s3 = __fmaf_rn(t3, t3, s3);
            }
            float m = 0.f;
            if (half == 0 && in) {
                const float rt = __fsqrt_rn(__fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2, s3)));
                const float v = __fmul_rn(rt, rt);
                m = s_m[i];
                if (v < m) s_m[i] = m = v;
            }
            if (ci > 1) group_sum(g, m);
        }
        if (ci == 1) {
            // the first draw's e, from the largest distance of all blocks
            __syncthreads();
            if (t < 32) {
                unsigned top = 0;  // floats >= 0 order as their bits
                for (int i = t; i < rows; i += 32) top = max(top, __float_as_uint(s_m[i]));
                top = __reduce_max_sync(0xffffffffu, top);
                unsigned long long *const maxs = words + 2 * (size_t)G + 4, v[SEED_SPAN];
                if (t == 0) seed_store(maxs + blockIdx.x, (unsigned long long)top << 2 | 1u);
                const bool ok = seed_gather(maxs, G, 1, s_words, v, err);
#pragma unroll
                for (int i = 0; i < SEED_SPAN; ++i) top = max(top, (unsigned)v[i]);
                top = __reduce_max_sync(0xffffffffu, top);
                // top < 2^(x - 126), so n of them stay below 2^(x - 126 + bits of n)
                if (t == 0) {
                    s_e = max((int)(top >> 23) - 126 + (64 - __clzll(n)) - 61, -149);
                    s_word = ok;
                }
            }
            __syncthreads();
            if (s_word == 0) return;
            e = s_e;
            for (int g = warp; g * 16 < rows; g += SEED_NT / 32) {
                const int i = g * 16 + (lane >> 1);
                group_sum(g, half == 0 && i < rows ? s_m[i] : 0.f);
            }
        }
        __syncthreads();
        if (t < 32) {
            int next_e = e;
            const unsigned bits = __float_as_uint(u[ci - 1]), x = bits >> 23;
            const unsigned long long w = seed_draw<16>(
                words + (size_t)(ci & 1) * G, words + 2 * (size_t)G + (ci & 1), ci, s_group, rows, b0, s_words,
                [&](int i) { return seed_fixed(s_m[i], e); },
                [&](unsigned long long total, unsigned long long &target, unsigned long long &band,
                    unsigned long long &) {
                    // u in 2^-64ths; u = 1 (rounded up by the generator's library): the total
                    const unsigned long long mant = (bits & 0x7fffffu) | 0x800000u;
                    const int shift = (int)x - 86;
                    const unsigned long long u64 = shift >= 0 ? mant << min(shift, 40) : mant >> min(-shift, 63);
                    target = x >= 127 ? total : __umul64hi(total, u64);
                    // 2 x 2 n 2^-53 total, and four rows' worth of the roundings to 2^e
                    band = __umul64hi(total, (unsigned long long)n << 13) + 4ull * (unsigned long long)n + 4ull;
                    // the next draw's total is below this one's and n more
                    next_e = max(e - max(__clzll((long long)(total + (unsigned long long)n)) - 3, 0), -149);
                    return true;
                },
                err);
            if (lane == 0) {
                s_word = w;
                s_e = next_e;
            }
        }
        __syncthreads();
        unsigned long long w = s_word;
        if (w == 0) return;  // a wait gave up (in every block, in the end)
        e = s_e;
        if (w & SEED_AGAIN) {
            ++again;
            for (int i = t; i < rows; i += SEED_NT) min_sq[b0 + i] = s_m[i];
            __threadfence();
            __syncthreads();
            unsigned long long *const serial = words + 2 * (size_t)G + 2 + (ci & 1);
            if (t == 0) {
                atomicAdd(done, 1u);
                bool ok = true;
                if (blockIdx.x == 0) {
                    unsigned polls = 0;
                    while (*reinterpret_cast<volatile unsigned *>(done) < again * (unsigned)G && ok)
                        ok = ++polls < SEED_SPINS;
                    __threadfence();
                    if (ok) {
                        w = (unsigned long long)ci << SEED_TAG | (unsigned long long)kpp_serial(min_sq, n, u[ci - 1]);
                        seed_store(serial, w);
                    } else {
                        *reinterpret_cast<volatile int *>(err) = 1;
                    }
                } else {
                    ok = seed_wait(serial, ci, &w, err, SEED_SPINS * 16u);
                }
                s_word = ok ? w : 0;
            }
            __syncthreads();
            w = s_word;
            if (w == 0) return;
        }
        const float *row = X + (int64_t)(w & (SEED_AGAIN - 1)) * dp;
        for (int j = t; j < dp; j += SEED_NT) {
            const float v = __ldg(row + j);
            s_c[j] = v;
            if (blockIdx.x == 0) C[(int64_t)ci * dp + j] = v;
        }
        __syncthreads();
    }
}

// ── row norms ─────────────────────────────────────────────────────────────
__global__ void row_norms_kernel(const float *__restrict__ X, int64_t n, int dp, float *__restrict__ out) {
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    float s = 0.f;
    for (int j = lane; j < dp; j += 32) {
        float v = X[row * dp + j];
        s = fmaf(v, v, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[row] = s;
}

// ── float assignment: tile GEMM + argmin ──────────────────────────────────
// The first nearest centroid of row x in f2ord's total order, by one warp: for rows with a
// product that is not finite (a NaN score has a place in that order, but none in
// AssignBest's compares) or without any score below +inf.
__device__ __noinline__ int32_t assign_unordered(const float *__restrict__ x, const float *__restrict__ C,
                                                 const float *__restrict__ cnorm, int k, int dp) {
    uint64_t best = KEY_EMPTY;
    for (int c = threadIdx.x & 31; c < k; c += 32) {
        float dot = 0.f;
        for (int j = 0; j < dp; ++j) dot = fmaf(x[j], C[(int64_t)c * dp + j], dot);
        const uint64_t key = make_key(f2ord(fmaf(-2.f, dot, cnorm[c])), (uint32_t)c);
        best = key < best ? key : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other < best ? other : best;
    }
    return (int32_t)key_idx(best);
}

// The nearest centroid so far of a warp's eight rows, over this lane's columns, which
// come in ascending order (a key of score and index per product took nine
// instructions, a compare and two selects take four with the score itself).
struct AssignBest {
    float v[8];
    int c[8];
    f32x2 sum[8];  // of the products: finite only if all of them are
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[i] = INFINITY;
            c[i] = 0;
            sum[i] = 0ull;
        }
    }
    // cn: |c|^2 of column gt_col(p) + e, +inf past the last
    template <int H, typename Norm>
    __device__ __forceinline__ void add(const f32x2 (&acc)[8][2 * H], int c0, Norm &&cn) {
#pragma unroll
        for (int p = 0; p < 2 * H; ++p) {
            const int col = c0 + gt_col(p);
#pragma unroll
            for (int i = 0; i < 8; ++i) sum[i] = add2(sum[i], acc[i][p]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float norm = cn(col + e);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float lo, hi;
                    unpack2(acc[i][p], lo, hi);
                    const float x = fmaf(-2.f, e ? hi : lo, norm);
                    const bool less = x < v[i];
                    v[i] = less ? x : v[i];
                    c[i] = less ? col + e : c[i];
                }
            }
        }
    }
    // the labels of rows p0 .. p0 + 7 (those below p1); adds up the changed ones
    __device__ __forceinline__ void finish(const float *__restrict__ X, int64_t p0, int64_t p1, int dp,
                                           const float *__restrict__ C, const float *__restrict__ cnorm, int k,
                                           int32_t *__restrict__ labels, unsigned long long *__restrict__ n_changed) {
        const int lane = threadIdx.x & 31;
        int32_t mine = 0;  // lane i: row i's label
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t o = f2ord(v[i]), top = __reduce_min_sync(0xffffffffu, o);
            int32_t lab = (int32_t)__reduce_min_sync(0xffffffffu, o == top ? (unsigned)c[i] : 0xffffffffu);
            float lo, hi;
            unpack2(sum[i], lo, hi);
            const bool odd = __any_sync(0xffffffffu, !(fabsf(lo) < INFINITY && fabsf(hi) < INFINITY));
            if ((odd || top >= f2ord(INFINITY)) && p0 + i < p1)
                lab = assign_unordered(X + (p0 + i) * dp, C, cnorm, k, dp);
            if (lane == i) mine = lab;
        }
        const bool changed = lane < 8 && p0 + lane < p1 && labels[p0 + lane] != mine;
        if (changed) labels[p0 + lane] = mine;
        const unsigned m = __ballot_sync(0xffffffffu, changed);
        if (lane == 0 && m) atomicAdd(n_changed, (unsigned long long)__popc(m));
    }
};

template <int H>
__global__ void __launch_bounds__(GT_THREADS, 2) kmeans_assign_kernel(const float *__restrict__ X, int64_t n, int dp,
                                                                      const float *__restrict__ C,
                                                                      const float *__restrict__ cnorm, int k,
                                                                      int32_t *__restrict__ labels,
                                                                      unsigned long long *__restrict__ n_changed) {
    extern __shared__ __align__(16) uint8_t gt_raw[];
    GemmTileSmem<H> &s = *reinterpret_cast<GemmTileSmem<H> *>(gt_raw);
    __shared__ int64_t arow[GT_BM];
    const int64_t p0 = (int64_t)blockIdx.x * GT_BM;
    if (threadIdx.x < GT_BM) arow[threadIdx.x] = (p0 + threadIdx.x < n) ? p0 + threadIdx.x : -1;
    __syncthreads();
    AssignBest best;
    best.init();
    f32x2 acc[8][2 * H];
    for (int c0 = 0; c0 < k; c0 += GT_BN * H) {
        gt_tile<H>(s, acc, X, arow, dp, C, c0, k, dp, dp);
        best.add<H>(acc, c0, [&](int c) { return c < k ? cnorm[c] : INFINITY; });
    }
    best.finish(X, p0 + (threadIdx.x >> 5) * 8, n, dp, C, cnorm, k, labels, n_changed);
}

// The same for centroids that fit shared memory beside a second block (128 H of them):
// a block keeps them there over a run of rows and reads nothing but rows, whose next
// slice is always in flight, also across tiles.  100k x 64 against 256 centroids: 92 us
// with the centroids read again for every 64 rows, 84 us here (45 us of FP32
// pipe).
constexpr size_t ASSIGN_SMEM_MAX = 110 * 1024;
template <int H>
static size_t assign_smem(int dp) {
    return (size_t)dp * (GT_BN * H + 4) * 4 + sizeof(GemmTileSmem<H>::As) + GT_BN * H * 4;
}
template <int H>
__global__ void __launch_bounds__(GT_THREADS, 2)
    kmeans_assign_resident_kernel(const float *__restrict__ X, int64_t n, int dp, const float *__restrict__ C,
                                  const float *__restrict__ cnorm, int k, int per_block,
                                  int32_t *__restrict__ labels, unsigned long long *__restrict__ n_changed) {
    extern __shared__ __align__(16) uint8_t gt_raw[];
    constexpr int BP = GT_BN * H + 4;
    float2(*As)[GT_BK][GT_BM + 2] = reinterpret_cast<float2(*)[GT_BK][GT_BM + 2]>(gt_raw);
    float *const Bs = reinterpret_cast<float *>(gt_raw + sizeof(GemmTileSmem<H>::As));  // [dp][BP]
    float *const s_cn = Bs + (size_t)dp * BP;
    const int t = threadIdx.x, tm = t >> 5, tn = t & 31;
    const int dp4 = dp >> 2, nk = dp / GT_BK;
    for (int i = t; i < GT_BN * H * dp4; i += GT_THREADS) {
        const int c = i / dp4, j = i % dp4;
        const float4 v = c < k ? __ldg(reinterpret_cast<const float4 *>(C + (int64_t)c * dp) + j)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        Bs[(4 * j + 0) * BP + c] = v.x;
        Bs[(4 * j + 1) * BP + c] = v.y;
        Bs[(4 * j + 2) * BP + c] = v.z;
        Bs[(4 * j + 3) * BP + c] = v.w;
    }
    for (int c = t; c < GT_BN * H; c += GT_THREADS) s_cn[c] = c < k ? cnorm[c] : INFINITY;
    const int64_t p0 = (int64_t)blockIdx.x * per_block, p1 = min(n, p0 + per_block);
    // this thread's float4 of each slice: row t / 4 of the tile, k 4 (t % 4) ..
    const int r = t >> 2, k4 = t & 3;
    float4 ra;
    auto load = [&](int64_t tile, int kc) {
        ra = tile + r < p1 ? __ldg(reinterpret_cast<const float4 *>(X + (tile + r) * dp) + kc * (GT_BK / 4) + k4)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto store = [&](int buf) {
        As[buf][4 * k4 + 0][r] = make_float2(ra.x, ra.x);
        As[buf][4 * k4 + 1][r] = make_float2(ra.y, ra.y);
        As[buf][4 * k4 + 2][r] = make_float2(ra.z, ra.z);
        As[buf][4 * k4 + 3][r] = make_float2(ra.w, ra.w);
    };
    if (p0 < p1) {
        load(p0, 0);
        store(0);
    }
    __syncthreads();
    int cur = 0;
    for (int64_t tile = p0; tile < p1; tile += GT_BM) {
        f32x2 acc[8][2 * H];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int p = 0; p < 2 * H; ++p) acc[i][p] = 0ull;
        const bool work = tile + tm * 8 < p1;  // else this warp has no rows in the last tile
        for (int kc = 0; kc < nk; ++kc, cur ^= 1) {
            const bool more = kc + 1 < nk || tile + GT_BM < p1;
            if (kc + 1 < nk) load(tile, kc + 1);
            else if (more) load(tile + GT_BM, 0);
            if (work) {
                const float *b = Bs + (size_t)kc * GT_BK * BP + tn * 4;
#pragma unroll
                for (int kk = 0; kk < GT_BK; ++kk) {
                    f32x2 av[8], bv[2 * H];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&As[cur][kk][tm * 8 + 2 * i]);
                        av[2 * i] = x.x;
                        av[2 * i + 1] = x.y;
                    }
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(b + kk * BP + h * GT_BN);
                        bv[2 * h] = x.x;
                        bv[2 * h + 1] = x.y;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int p = 0; p < 2 * H; ++p) acc[i][p] = fma2(av[i], bv[p], acc[i][p]);
                }
            }
            if (more) store(cur ^ 1);
            __syncthreads();
        }
        if (!work) continue;
        AssignBest best;
        best.init();
        best.add<H>(acc, 0, [&](int c) { return s_cn[c]; });
        best.finish(X, tile + tm * 8, p1, dp, C, cnorm, k, labels, n_changed);
    }
}

// ── float update: FP64 sums ───────────────────────────────────────────────
// (this kernel and the next do nothing when no label changed, so that the host
// can launch a whole iteration before it reads the change count)
__global__ void kmeans_accumulate_kernel(const float *__restrict__ X, int64_t n, int d, int dp,
                                         const int32_t *__restrict__ labels,
                                         const unsigned long long *__restrict__ n_changed, double *__restrict__ sums,
                                         int64_t *__restrict__ counts) {
    if (*n_changed == 0) return;
    const int64_t p = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (p >= n) return;
    const int32_t c = labels[p];
    if (lane == 0) atomicAdd(reinterpret_cast<unsigned long long *>(counts + c), 1ull);
    for (int j = lane; j < d; j += 32) atomicAdd(sums + (int64_t)c * dp + j, (double)X[p * dp + j]);
}

__global__ void kmeans_finalize_kernel(const double *__restrict__ sums, const int64_t *__restrict__ counts, int k,
                                       int d, int dp, const unsigned long long *__restrict__ n_changed,
                                       float *__restrict__ C) {
    if (*n_changed == 0) return;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)k * dp) return;
    const int c = (int)(t / dp), j = (int)(t % dp);
    if (counts[c] > 0) C[t] = (j < d) ? (float)(sums[t] / (double)counts[c]) : 0.f;
}

int kmeans_l2_device(const float *X, int64_t n, int d, int dp, int64_t k, int64_t max_iter, uint32_t seed,
                     float *C, float *cnorm, int32_t *labels, int64_t *iters_out, cudaStream_t st) {
    if (dp % GT_BK) return fail(GN_ERR_INVALID, "kmeans: row stride must be a multiple of 16 floats");
    std::mt19937 rng(seed);
    std::uniform_int_distribution<size_t> pick_point(0, (size_t)n - 1);
    std::uniform_real_distribution<float> unif01(0.f, 1.f);
    const size_t row_bytes = (size_t)dp * sizeof(float);

    // k-means++ seeding, all on the device: the reference's draws (the first
    // point, then one uniform per further centroid) do not depend on the data,
    // so they are taken from the mt19937 stream up front in the reference's
    // order; each further centroid is one kpp_kernel launch, or all of them one
    // kpp_seed_kernel launch where the rows fit the SMs' shared memory
    GN_CUDA_TRY(cudaMemcpyAsync(C, X + pick_point(rng) * dp, row_bytes, cudaMemcpyDeviceToDevice, st));
    DBuf dmin, dpart, ddone;
    const int64_t chunk = round_up(ceil_div(n, KPP_NT * KPP_SPAN), KPP_ROWS);
    const int P = (int)ceil_div(n, chunk);
    if (k > 1) {
        GN_TRY(dmin.ensure((size_t)n * sizeof(float)));
        GN_TRY(dpart.ensure((size_t)P * sizeof(double)));
        GN_TRY(ddone.ensure(sizeof(unsigned)));
        GN_CUDA_TRY(cudaMemsetAsync(ddone.p, 0, sizeof(unsigned), st));
    }
    std::vector<float> us((size_t)std::max<int64_t>(k - 1, 0));
    for (float &v : us) v = unif01(rng);
    const int G = dev_info().num_sms;
    const int64_t seed_chunk = ceil_div(n, G);
    const size_t seed_smem = ((size_t)dp + round_up(seed_chunk, 16) + (size_t)seed_chunk * (dp + 8)) * 4 +
                             (size_t)ceil_div(seed_chunk, 32) * 16;
    DBuf dus, dwords;  // dwords: the blocks' words, then the arrivals and the error word
    const bool seeded = k > 1 && k < (1 << 23) && G <= 32 * SEED_SPAN && seed_smem <= SEED_SMEM_MAX;
    if (seeded) {
        const size_t words = 3 * (size_t)G + 4;
        GN_TRY(dus.ensure(us.size() * sizeof(float)));
        GN_TRY(dwords.ensure((words + 1) * 8));
        GN_CUDA_TRY(cudaMemcpyAsync(dus.p, us.data(), us.size() * sizeof(float), cudaMemcpyHostToDevice, st));
        GN_CUDA_TRY(cudaMemsetAsync(dwords.p, 0, (words + 1) * 8, st));
        GN_CUDA_TRY(cudaFuncSetAttribute(kpp_seed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)SEED_SMEM_MAX));
        unsigned long long *dw = dwords.as<unsigned long long>();
        unsigned *arrived = reinterpret_cast<unsigned *>(dw + words);
        int *derr = reinterpret_cast<int *>(dw + words) + 1, ki = (int)k, chunk_i = (int)seed_chunk;
        const float *du = dus.as<float>();
        float *dm = dmin.as<float>();
        void *args[] = {&X, &n, &d, &dp, &C, &ki, &du, &dm, &chunk_i, &dw, &arrived, &derr};
        GN_CUDA_TRY(cudaLaunchCooperativeKernel((void *)kpp_seed_kernel, dim3(G), dim3(SEED_NT), args, seed_smem, st));
        int herr = 0;
        GN_CUDA_TRY(cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, st));
        GN_CUDA_TRY(cudaStreamSynchronize(st));
        if (herr) return fail(GN_ERR_TIMEOUT, "kmeans: a wait of the seeding ran out");
    } else {
        for (int64_t ci = 1; ci < k; ++ci)
            kpp_kernel<<<(unsigned)P, KPP_NT, 0, st>>>(X, n, d, dp, C, ci, us[(size_t)ci - 1], dmin.as<float>(), chunk,
                                                       P, dpart.as<double>(), ddone.as<unsigned>());
    }
    GN_CUDA_TRY(cudaGetLastError());

    // Lloyd iterations; one host synchronisation each (the change count and the
    // cluster sizes together)
    DBuf dsum, dstat;
    GN_TRY(dsum.ensure((size_t)k * dp * sizeof(double)));
    // change count, then rows per cluster, 256 bytes on: the counts' atomics would hold up the
    // blocks that read the change count next to them (300,000 rows of one coordinate, 10
    // clusters: 219 us an update, 183 so)
    constexpr int64_t STAT_AT = 32;
    GN_TRY(dstat.ensure((size_t)(k + STAT_AT) * sizeof(int64_t)));
    unsigned long long *dchg = dstat.as<unsigned long long>();
    int64_t *dcnt = dstat.as<int64_t>() + STAT_AT;
    GN_CUDA_TRY(cudaMemsetAsync(labels, 0, (size_t)n * sizeof(int32_t), st));
    std::vector<int64_t> hstat((size_t)(k + STAT_AT));
    GN_CUDA_TRY(cudaFuncSetAttribute(kmeans_assign_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(GemmTileSmem<2>)));
    GN_CUDA_TRY(cudaFuncSetAttribute(kmeans_assign_resident_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)ASSIGN_SMEM_MAX));
    GN_CUDA_TRY(cudaFuncSetAttribute(kmeans_assign_resident_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)ASSIGN_SMEM_MAX));
    // two blocks per SM, each with an equal run of rows (whole warps' eights)
    const int64_t per_block = std::max<int64_t>(round_up(ceil_div(n, 2 * (int64_t)G), 8), GT_BM);
    const unsigned blocks = (unsigned)ceil_div(n, per_block), tiles = (unsigned)ceil_div(n, GT_BM);
    auto assign = [&]() {
        if (k <= GT_BN && assign_smem<1>(dp) <= ASSIGN_SMEM_MAX && per_block < (1 << 30))
            kmeans_assign_resident_kernel<1><<<blocks, GT_THREADS, assign_smem<1>(dp), st>>>(
                X, n, dp, C, cnorm, (int)k, (int)per_block, labels, dchg);
        else if (k > GT_BN && k <= 2 * GT_BN && assign_smem<2>(dp) <= ASSIGN_SMEM_MAX && per_block < (1 << 30))
            kmeans_assign_resident_kernel<2><<<blocks, GT_THREADS, assign_smem<2>(dp), st>>>(
                X, n, dp, C, cnorm, (int)k, (int)per_block, labels, dchg);
        else if (k <= GT_BN)
            kmeans_assign_kernel<1><<<tiles, GT_THREADS, sizeof(GemmTileSmem<1>), st>>>(X, n, dp, C, cnorm, (int)k,
                                                                                        labels, dchg);
        else
            kmeans_assign_kernel<2><<<tiles, GT_THREADS, sizeof(GemmTileSmem<2>), st>>>(X, n, dp, C, cnorm, (int)k,
                                                                                        labels, dchg);
    };
    int64_t it = 0;
    for (; it < max_iter; ++it) {
        row_norms_kernel<<<(unsigned)ceil_div(k, 8), 256, 0, st>>>(C, k, dp, cnorm);
        GN_CUDA_TRY(cudaMemsetAsync(dstat.p, 0, hstat.size() * sizeof(int64_t), st));
        GN_CUDA_TRY(cudaMemsetAsync(dsum.p, 0, (size_t)k * dp * sizeof(double), st));
        assign();
        kmeans_accumulate_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, st>>>(X, n, d, dp, labels, dchg,
                                                                          dsum.as<double>(), dcnt);
        kmeans_finalize_kernel<<<(unsigned)ceil_div(k * dp, 256), 256, 0, st>>>(dsum.as<double>(), dcnt, (int)k, d, dp,
                                                                              dchg, C);
        GN_CUDA_TRY(cudaMemcpyAsync(hstat.data(), dstat.p, hstat.size() * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        GN_CUDA_TRY(cudaStreamSynchronize(st));
        if (hstat[0] == 0) break;
        for (int64_t c = 0; c < k; ++c)
            if (hstat[(size_t)(c + STAT_AT)] == 0)
                GN_CUDA_TRY(cudaMemcpyAsync(C + c * dp, X + pick_point(rng) * dp, row_bytes,
                                            cudaMemcpyDeviceToDevice, st));
    }
    row_norms_kernel<<<(unsigned)ceil_div(k, 8), 256, 0, st>>>(C, k, dp, cnorm);
    GN_CUDA_TRY(cudaGetLastError());
    if (iters_out) *iters_out = it;
    return GN_OK;
}

void row_norms(const float *X, int64_t n, int dp, float *out, cudaStream_t st) {
    if (n > 0) row_norms_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, st>>>(X, n, dp, out);
}

// ── binary k-means ────────────────────────────────────────────────────────
// This thread's KPP_SPAN neighbouring sums of the P chunks, and their total.
__device__ __forceinline__ int64_t bin_span(const int64_t *sums, int P, int64_t (&ps)[KPP_SPAN]) {
#pragma unroll
    for (int i = 0; i < KPP_SPAN; ++i) {
        const int p = threadIdx.x * KPP_SPAN + i;
        ps[i] = p < P ? __ldcg(sums + p) : 0;
    }
    return (ps[0] + ps[1]) + (ps[2] + ps[3]);
}

// The point of the running sums: the first index i with min_d[0] + .. +
// min_d[i] > r (0 <= r < total), exact in int64, by one block: sums holds the
// sums of P chunks of `chunk` rows, pre this thread's running sum before its
// KPP_SPAN sums ps.  Writes row i of X to C[ci].
__device__ __forceinline__ void bin_pick(const uint4 *__restrict__ X, int64_t n, int w4, uint4 *C, int64_t ci,
                                         const int32_t *min_d, int64_t chunk, const int64_t (&ps)[KPP_SPAN],
                                         int64_t r, int64_t pre) {
    __shared__ int s_chunk;
    __shared__ int64_t s_before, s_row;
    const int t = threadIdx.x;
    if (t == 0) {  // in range whatever r is
        s_chunk = 0;
        s_before = 0;
        s_row = 0;
    }
    __syncthreads();
    int64_t cum = pre;
#pragma unroll
    for (int i = 0; i < KPP_SPAN; ++i) {  // sums are not negative: exactly one chunk takes the running sum past r
        if (cum <= r && cum + ps[i] > r) {
            s_chunk = t * KPP_SPAN + i;
            s_before = cum;
        }
        cum += ps[i];
    }
    __syncthreads();
    const int64_t c0 = (int64_t)s_chunk * chunk, c1 = min(n, c0 + chunk);
    const int64_t per = (c1 - c0 + KPP_NT - 1) / KPP_NT;
    const int64_t e0 = min(c1, c0 + t * per), e1 = min(c1, e0 + per);
    int64_t ls = 0, lt;
    for (int64_t i = e0; i < e1; ++i) ls += __ldcg(min_d + i);
    cum = s_before + kpp_block_scan(ls, &lt);
    for (int64_t i = e0; i < e1; ++i) {
        const int64_t v = per == 1 ? ls : __ldcg(min_d + i);
        if (cum <= r && cum + v > r) s_row = i;
        cum += v;
    }
    __syncthreads();
    const int64_t row = s_row;
    for (int j = t; j < w4; j += KPP_NT) C[ci * w4 + j] = X[row * w4 + j];
}

// std::uniform_int_distribution's value in [0, range) from a stream of 32-bit
// generator outputs: Lemire's multiply-and-reject method (ACM TOMACS 29(1),
// 2019), which libstdc++ uses for ranges that fit 32 bits.  Takes outputs from
// raw at *cur; a stream that runs out leaves *cur past nraw.
__device__ __forceinline__ uint32_t bin_draw(const uint32_t *__restrict__ raw, int nraw, int *cur, uint32_t range) {
    uint64_t prod = (uint64_t)(*cur < nraw ? raw[*cur] : 0u) * range;
    ++*cur;
    if ((uint32_t)prod < range) {
        const uint32_t floor = (0u - range) % range;
        while ((uint32_t)prod < floor && *cur < nraw) {
            prod = (uint64_t)raw[*cur] * range;
            ++*cur;
        }
    }
    return (uint32_t)(prod >> 32);
}

// One launch per draw of the binary k-means++ (BinaryIVF.hpp:140-170): every
// block lowers its chunk's distances by the newest centroid (row ci - 1) and
// sums the chunk; the last block to finish draws centroid ci as the reference
// does: pick(rng), then, when the total is positive, r = wsel(rng) in
// [0, total) and the first row whose running sum passes r.  The generator's
// outputs come from raw at *cursor (the host moves its generator on by what
// was used).  raw == NULL: the last block only writes the total, and the host
// draws (bin_pick_kernel follows).
// 200k x 32 bytes, 255 draws: 58.6 ms with one thread walking the sums and two
// host round trips per draw, 2.4 ms as one launch each.
__global__ void __launch_bounds__(KPP_NT) bin_kpp_kernel(const uint4 *__restrict__ X, int64_t n, int w4, uint4 *C,
                                                         int64_t ci, int32_t *min_d, int64_t chunk, int P,
                                                         int64_t *sums, unsigned *done,
                                                         const uint32_t *__restrict__ raw, int nraw, int *cursor,
                                                         int64_t *total_out) {
    const int t = threadIdx.x;
    const int64_t b0 = (int64_t)blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    const uint4 *c = C + (ci - 1) * w4;
    int64_t s = 0, tot;
    for (int64_t i = b0 + t; i < b1; i += KPP_NT) {
        const int32_t v = (int32_t)hdist(c, X + i * w4, w4);
        int32_t m = v;
        if (ci > 1) m = min(v, min_d[i]);
        min_d[i] = m;
        s += m;
    }
    kpp_block_scan(s, &tot);
    if (t == 0) sums[blockIdx.x] = tot;
    if (!kpp_last_block(done)) return;

    int64_t ps[KPP_SPAN], total;
    const int64_t pre = kpp_block_scan(bin_span(sums, P, ps), &total);
    if (!raw) {
        if (t == 0) *total_out = total;
        return;
    }
    __shared__ int64_t s_r, s_first;
    if (t == 0) {
        int cur = *cursor;
        s_first = bin_draw(raw, nraw, &cur, (uint32_t)n);
        s_r = -1;
        if (total > 0) s_r = (int64_t)bin_draw(raw, nraw, &cur, (uint32_t)total);
        *cursor = cur;
    }
    __syncthreads();
    if (s_r >= 0) {
        bin_pick(X, n, w4, C, ci, min_d, chunk, ps, s_r, pre);
    } else {  // every row equals a centroid: the first draw stands
        for (int j = t; j < w4; j += KPP_NT) C[ci * w4 + j] = X[s_first * w4 + j];
    }
}

// The binary draws in one launch (see kpp_seed_kernel): bin_kpp_kernel's draws, which
// every block makes for itself from the generator's outputs, since it reads all the
// sums.  words: [2][grid] sums, then [2] rows, zeroed; *cursor: outputs used.
__global__ void __launch_bounds__(SEED_NT, 1) bin_seed_kernel(const uint4 *__restrict__ X, int64_t n, int w4, uint4 *C,
                                                              int k, int chunk, unsigned long long *words,
                                                              const uint32_t *__restrict__ raw, int nraw, int *cursor,
                                                              int *err) {
    extern __shared__ __align__(16) uint4 bseed_smem[];
    __shared__ unsigned long long s_word, s_words[32 * SEED_SPAN];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, G = gridDim.x;
    const int64_t b0 = min(n, (int64_t)blockIdx.x * chunk);
    const int rows = (int)(min(n, b0 + chunk) - b0);
    const int stride = w4 | 1;  // odd: neighbouring rows in different banks
    uint4 *const s_c = bseed_smem, *const s_x = s_c + w4;
    unsigned long long *const s_group = reinterpret_cast<unsigned long long *>(s_x + (size_t)chunk * stride);
    uint32_t *const s_m = reinterpret_cast<uint32_t *>(s_group + (chunk + 31) / 32);
    for (int i = t; i < rows * w4; i += SEED_NT) s_x[(i / w4) * stride + i % w4] = ldg_nc_u4(X + b0 * w4 + i);
    for (int i = t; i < rows; i += SEED_NT) s_m[i] = 0xffffffffu;
    for (int j = t; j < w4; j += SEED_NT) s_c[j] = C[j];
    __syncthreads();
    int cur = 0;
    for (int ci = 1; ci < k; ++ci) {
        for (int g = warp; g * 32 < rows; g += SEED_NT / 32) {
            const int i = g * 32 + lane;
            uint32_t m = 0;
            if (i < rows) s_m[i] = m = min(s_m[i], (uint32_t)hdist(s_c, s_x + i * stride, w4));
            m = __reduce_add_sync(0xffffffffu, m);
            if (lane == 0) s_group[g] = m;
        }
        __syncthreads();
        if (t < 32) {
            const unsigned long long w = seed_draw<32>(
                words + (size_t)(ci & 1) * G, words + 2 * (size_t)G + (ci & 1), ci, s_group, rows, b0, s_words,
                [&](int i) { return (unsigned long long)s_m[i]; },
                [&](unsigned long long total, unsigned long long &target, unsigned long long &band,
                    unsigned long long &word) {
                    // every row equals a centroid: the first draw stands
                    word = (unsigned long long)ci << SEED_TAG | bin_draw(raw, nraw, &cur, (uint32_t)n);
                    if (total == 0) return false;
                    target = 1ull + bin_draw(raw, nraw, &cur, (uint32_t)total);  // the running sum passes the draw
                    band = 0;
                    return true;
                },
                err);
            if (lane == 0) s_word = w;
        }
        __syncthreads();
        const unsigned long long w = s_word;
        if (w == 0) return;  // a wait gave up (in every block, in the end)
        const uint4 *row = X + (int64_t)(w & (SEED_AGAIN - 1)) * w4;
        for (int j = t; j < w4; j += SEED_NT) {
            const uint4 v = ldg_nc_u4(row + j);
            s_c[j] = v;
            if (blockIdx.x == 0) C[(int64_t)ci * w4 + j] = v;
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && t == 0) *cursor = cur;
}

// The pick for an r that the host drew.
__global__ void __launch_bounds__(KPP_NT) bin_pick_kernel(const uint4 *__restrict__ X, int64_t n, int w4, uint4 *C,
                                                          int64_t ci, const int32_t *min_d, int64_t chunk, int P,
                                                          const int64_t *sums, int64_t r) {
    int64_t ps[KPP_SPAN], total;
    const int64_t pre = kpp_block_scan(bin_span(sums, P, ps), &total);
    bin_pick(X, n, w4, C, ci, min_d, chunk, ps, r, pre);
}

// assignment to the first nearest centroid; centroids staged in shared memory
__global__ void bin_assign_kernel(const uint4 *__restrict__ X, int64_t n, int w4, const uint4 *__restrict__ C, int k,
                                  int32_t *__restrict__ labels, unsigned long long *__restrict__ n_changed) {
    extern __shared__ uint4 sc[];
    for (int i = threadIdx.x; i < k * w4; i += blockDim.x) sc[i] = C[i];
    __syncthreads();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool changed = false;
    if (p < n) {
        uint32_t best = 0xffffffffu;
        int32_t bc = 0;
        const uint4 *x = X + p * w4;
        if (w4 == 4) {
            const uint4 x0 = x[0], x1 = x[1], x2 = x[2], x3 = x[3];
            for (int c = 0; c < k; ++c) {
                const uint4 *cc = sc + c * 4;
                const uint32_t dd = popc8(x0, cc[0], x1, cc[1]) + popc8(x2, cc[2], x3, cc[3]);
                if (dd < best) { best = dd; bc = c; }
            }
        } else if (w4 == 2) {
            const uint4 x0 = x[0], x1 = x[1];
#pragma unroll 4
            for (int c = 0; c < k; ++c) {
                const uint32_t dd = popc8(x0, sc[2 * c], x1, sc[2 * c + 1]);
                if (dd < best) { best = dd; bc = c; }
            }
        } else {
            for (int c = 0; c < k; ++c) {
                const uint32_t dd = hdist(x, sc + c * w4, w4);
                if (dd < best) { best = dd; bc = c; }
            }
        }
        if (labels[p] != bc) { labels[p] = bc; changed = true; }
    }
    const unsigned m = __ballot_sync(0xffffffffu, changed);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(n_changed, (unsigned long long)__popc(m));
}

// Bit counts per cluster.  Block (x, y, z): a chunk of rows, 32-bit word y of
// each, clusters [z * BC_SLAB, ..).  A row adds its word to its cluster's 32
// shared counters as 16 atomic additions of two 16-bit counters each (bits b
// and b + 16; a chunk has at most BC_ROWS < 65536 rows), and the block adds
// its totals to the global counts once: 200k x 256 bits, 256 clusters: one
// global atomic per set bit took 208 us, this 18 us.
constexpr int BC_SLAB = 1024, BC_ROWS = 8192, BC_NT = 512;
__global__ void __launch_bounds__(BC_NT) bin_bitcount_kernel(const uint32_t *__restrict__ X, int64_t n, int w32,
                                                             int rows, const int32_t *__restrict__ labels, int k,
                                                             const unsigned long long *__restrict__ n_changed,
                                                             int32_t *__restrict__ counts, int32_t *__restrict__ cc) {
    extern __shared__ uint32_t bc[];  // [16][slab]: cluster c's pair j at bc[j * slab + c]; then, word 0, [slab] rows
    if (*n_changed == 0) return;
    const int slab0 = blockIdx.z * BC_SLAB, slab = min(BC_SLAB, k - slab0);
    const int w = blockIdx.y;
    const int words = slab * (w == 0 ? 17 : 16);
    for (int i = threadIdx.x; i < words; i += BC_NT) bc[i] = 0;
    __syncthreads();
    const int64_t r0 = (int64_t)blockIdx.x * rows, r1 = min(n, r0 + rows);
    for (int64_t p = r0 + threadIdx.x; p < r1; p += BC_NT) {
        const int c = labels[p] - slab0;
        if (c < 0 || c >= slab) continue;
        const uint32_t bits = X[p * w32 + w];
#pragma unroll
        for (int j = 0; j < 16; ++j) atomicAdd(bc + j * slab + c, (bits >> j) & 0x00010001u);
        if (w == 0) atomicAdd(bc + 16 * slab + c, 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < slab * 32; i += BC_NT) {
        const int c = i >> 5, b = i & 31;
        const uint32_t v = (bc[(b & 15) * slab + c] >> (b & 16)) & 0xffffu;
        if (v) atomicAdd(counts + ((int64_t)(slab0 + c) * w32 + w) * 32 + b, (int32_t)v);
    }
    if (w == 0)
        for (int c = threadIdx.x; c < slab; c += BC_NT)
            if (const uint32_t v = bc[16 * slab + c]) atomicAdd(cc + slab0 + c, (int32_t)v);
}

// majority vote (count > n_c / 2), a warp per word of a centroid; clusters with
// no point are left for the host, and so is everything when no label changed
__global__ void bin_majority_kernel(const int32_t *__restrict__ counts, const int32_t *__restrict__ cc, int64_t words,
                                    int w32, const unsigned long long *__restrict__ n_changed,
                                    uint32_t *__restrict__ C) {
    const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= words || *n_changed == 0) return;
    const int32_t m = cc[t / w32];
    if (m == 0) return;
    const uint32_t word = __ballot_sync(0xffffffffu, counts[t * 32 + (threadIdx.x & 31)] > m / 2);
    if ((threadIdx.x & 31) == 0) C[t] = word;
}

int kmeans_bin_device(const uint8_t *X, int64_t n, int nbytes, int w4, int32_t k, int32_t max_iter, uint32_t seed,
                      uint8_t *C, int32_t *labels, cudaStream_t st) {
    std::mt19937 rng(seed);
    std::uniform_int_distribution<size_t> pick(0, (size_t)n - 1);
    const size_t row = (size_t)w4 * 16;
    const uint4 *X4 = reinterpret_cast<const uint4 *>(X);
    GN_CUDA_TRY(cudaMemcpyAsync(C, X + pick(rng) * row, row, cudaMemcpyDeviceToDevice, st));
    DBuf dmin, dsums, daux, draw;
    const int64_t chunk = round_up(ceil_div(n, KPP_NT * KPP_SPAN), KPP_NT);
    const int P = (int)ceil_div(n, chunk);
    GN_TRY(dmin.ensure((size_t)n * 4));
    GN_TRY(dsums.ensure((size_t)P * 8));
    GN_TRY(daux.ensure(24));  // [0] total (int64), [2] arrival counter, [3] stream cursor, [4] error word
    GN_CUDA_TRY(cudaMemsetAsync(daux.p, 0, 24, st));
    int64_t *dtotal = daux.as<int64_t>();
    unsigned *ddone = daux.as<unsigned>() + 2;
    int *dcur = daux.as<int>() + 3;
    uint4 *C4 = reinterpret_cast<uint4 *>(C);
    // Every range below 2^32 (the rows, and the distances' total, at most n
    // rows x nbytes * 8 bits): the draws run on the device from the generator's
    // next outputs.  A draw takes two outputs and, rarely, more (each is
    // rejected with a probability below 1/2); 8 per centroid are on hand, and if
    // they should not do, the host draws instead, as for larger ranges.
#if defined(_GLIBCXX_RELEASE) && _GLIBCXX_RELEASE >= 11
    bool on_device = (uint64_t)n * (uint64_t)nbytes * 8 < (1ull << 32);
#else
    bool on_device = false;  // another library's distribution may draw differently
#endif
    if (on_device && k > 1) {
        std::vector<uint32_t> raw((size_t)k * 8 + 256);
        std::mt19937 ahead = rng;
        for (uint32_t &v : raw) v = (uint32_t)ahead();
        GN_TRY(draw.ensure(raw.size() * 4));
        GN_CUDA_TRY(cudaMemcpyAsync(draw.p, raw.data(), raw.size() * 4, cudaMemcpyHostToDevice, st));
        const int G = dev_info().num_sms;
        const int64_t seed_chunk = ceil_div(n, G);
        const size_t seed_smem =
            ((size_t)w4 + (size_t)seed_chunk * (w4 | 1)) * 16 + (size_t)ceil_div(seed_chunk, 32) * 8 + (size_t)seed_chunk * 4;
        DBuf dwords;
        int used[2] = {0, 0};  // outputs used, error word
        if (k < (1 << 23) && G <= 32 * SEED_SPAN && seed_smem <= SEED_SMEM_MAX) {
            const size_t words = 2 * (size_t)G + 2;
            GN_TRY(dwords.ensure(words * 8));
            GN_CUDA_TRY(cudaMemsetAsync(dwords.p, 0, words * 8, st));
            GN_CUDA_TRY(cudaFuncSetAttribute(bin_seed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)SEED_SMEM_MAX));
            unsigned long long *dw = dwords.as<unsigned long long>();
            int chunk_i = (int)seed_chunk, nraw = (int)raw.size(), *derr = dcur + 1;
            const uint32_t *dr = draw.as<uint32_t>();
            void *args[] = {&X4, &n, &w4, &C4, &k, &chunk_i, &dw, &dr, &nraw, &dcur, &derr};
            GN_CUDA_TRY(cudaLaunchCooperativeKernel((void *)bin_seed_kernel, dim3(G), dim3(SEED_NT), args, seed_smem,
                                                    st));
        } else {
            for (int32_t ci = 1; ci < k; ++ci)
                bin_kpp_kernel<<<(unsigned)P, KPP_NT, 0, st>>>(X4, n, w4, C4, ci, dmin.as<int32_t>(), chunk, P,
                                                               dsums.as<int64_t>(), ddone, draw.as<uint32_t>(),
                                                               (int)raw.size(), dcur, dtotal);
        }
        GN_CUDA_TRY(cudaMemcpyAsync(used, dcur, 8, cudaMemcpyDeviceToHost, st));
        GN_CUDA_TRY(cudaStreamSynchronize(st));
        if (used[1]) return fail(GN_ERR_TIMEOUT, "kmeans: a wait of the seeding ran out");
        on_device = used[0] <= (int)raw.size() - 1;
        if (on_device) rng.discard((unsigned long long)used[0]);
    }
    if (!on_device)
        for (int32_t ci = 1; ci < k; ++ci) {
            bin_kpp_kernel<<<(unsigned)P, KPP_NT, 0, st>>>(X4, n, w4, C4, ci, dmin.as<int32_t>(), chunk, P,
                                                           dsums.as<int64_t>(), ddone, nullptr, 0, dcur, dtotal);
            int64_t total = 0;
            GN_CUDA_TRY(cudaMemcpyAsync(&total, dtotal, 8, cudaMemcpyDeviceToHost, st));
            GN_CUDA_TRY(cudaStreamSynchronize(st));
            const size_t chosen = pick(rng);
            if (total > 0) {
                std::uniform_int_distribution<int64_t> wsel(0, total - 1);
                bin_pick_kernel<<<1, KPP_NT, 0, st>>>(X4, n, w4, C4, ci, dmin.as<int32_t>(), chunk, P,
                                                      dsums.as<int64_t>(), wsel(rng));
            } else {
                GN_CUDA_TRY(cudaMemcpyAsync(C + (size_t)ci * row, X + chosen * row, row, cudaMemcpyDeviceToDevice, st));
            }
        }

    // Lloyd iterations; one host synchronisation each (the change count and the
    // cluster sizes together): the update's kernels do nothing when no label changed
    const int w32 = w4 * 4;
    DBuf dcounts, dstat;
    GN_TRY(dcounts.ensure((size_t)k * w32 * 32 * 4));
    GN_TRY(dstat.ensure(8 + (size_t)k * 4));  // change count, then rows per cluster
    unsigned long long *dchg = dstat.as<unsigned long long>();
    int32_t *dcc = dstat.as<int32_t>() + 2;
    GN_CUDA_TRY(cudaMemsetAsync(labels, 0, (size_t)n * 4, st));
    const size_t smem = (size_t)k * row;
    if (smem > (size_t)dev_info().max_smem_optin)
        return fail(GN_ERR_UNSUPPORTED, "binary k-means: nlist * row bytes exceeds shared memory");
    if (smem > 48 * 1024)
        GN_CUDA_TRY(cudaFuncSetAttribute(bin_assign_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const size_t bc_smem = (size_t)std::min(k, BC_SLAB) * 17 * 4;
    if (bc_smem > 48 * 1024)
        GN_CUDA_TRY(cudaFuncSetAttribute(bin_bitcount_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bc_smem));
    const int slabs = (int)ceil_div(k, BC_SLAB);
    // rows per counting block: about two blocks per SM over the words and slabs
    const int64_t row_blocks = std::max<int64_t>(1, 2LL * dev_info().num_sms / ((int64_t)w32 * slabs));
    const int bc_rows = (int)std::min<int64_t>(BC_ROWS, std::max<int64_t>(BC_NT, ceil_div(n, row_blocks)));
    const dim3 bc_grid((unsigned)ceil_div(n, bc_rows), (unsigned)w32, (unsigned)slabs);
    std::vector<int32_t> hstat((size_t)k + 2);
    for (int32_t it = 0; it < max_iter; ++it) {
        GN_CUDA_TRY(cudaMemsetAsync(dstat.p, 0, 8 + (size_t)k * 4, st));
        GN_CUDA_TRY(cudaMemsetAsync(dcounts.p, 0, (size_t)k * w32 * 32 * 4, st));
        bin_assign_kernel<<<(unsigned)ceil_div(n, 256), 256, smem, st>>>(X4, n, w4, C4, k, labels, dchg);
        bin_bitcount_kernel<<<bc_grid, BC_NT, bc_smem, st>>>(reinterpret_cast<const uint32_t *>(X), n, w32, bc_rows,
                                                             labels, k, dchg, dcounts.as<int32_t>(), dcc);
        bin_majority_kernel<<<(unsigned)ceil_div((int64_t)k * w32, 8), 256, 0, st>>>(
            dcounts.as<int32_t>(), dcc, (int64_t)k * w32, w32, dchg, reinterpret_cast<uint32_t *>(C));
        GN_CUDA_TRY(cudaMemcpyAsync(hstat.data(), dstat.p, hstat.size() * 4, cudaMemcpyDeviceToHost, st));
        GN_CUDA_TRY(cudaStreamSynchronize(st));
        if (hstat[0] == 0 && hstat[1] == 0) break;
        for (int32_t c = 0; c < k; ++c)
            if (hstat[(size_t)c + 2] == 0)
                GN_CUDA_TRY(cudaMemcpyAsync(C + (size_t)c * row, X + pick(rng) * row, row, cudaMemcpyDeviceToDevice, st));
    }
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

}  // namespace gn
