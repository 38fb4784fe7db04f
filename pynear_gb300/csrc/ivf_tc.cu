// ivf_tc.cu — tensor-core engine of the float IVF index.
//
//   0. probes  coarse_probe_kernel: BF16 centroid scores (tc_ivf_kernel over
//              the centroids), the 64 best by counting, exact FP32
//              distances, then the first n_probe or the learned prober's
//              choice (its MLP fused here; from 1,024 queries the whole of it
//              runs in mlp_probe_kernel over 8 queries per block), and
//              each query's score bound for the scan;
//   1. plan    the same bucketing and work plan as the FP32 scan (ivf.cu),
//              score segments in 128-row slots;
//   2. Qb      the BF16 copy of each (query, probe) pair's query, rows grouped by
//              list (bucket order), so one TMA box covers a work unit's queries;
//   3. units   one tensor-core work unit per (list, row chunk, 128-query chunk);
//   4. scan    tc_ivf_kernel: BF16 tcgen05 GEMM of the list's rows (M = 128
//              per tile) against the unit's queries (N = 32..128) with FP32
//              accumulation; the minimum score |x|^2 - 2 q.x (exact FP32
//              |x|^2) of every 32-row quarter goes to the slot's four minima,
//              and the quarter's scores to the pair's slots when that minimum
//              is within the query's bound;
//   5. select  per query: a threshold from the quarter minima, only the
//              quarters below it are read, the S best keys (S = shortlist) by
//              counting, their squared L2 recomputed exactly in FP32 with a
//              compensated sum, the k nearest returned, ties to the lower
//              original index.
// Work units are short (a list holds ~1k rows), so selection is kept out of
// the tensor-core kernel: a per-unit top-S would pay its warm-up on every
// unit.  Everything stays on the device; the batch has no host round trip.
#include <cuda_bf16.h>

#include <algorithm>
#include <vector>

#include "f32x2.cuh"
#include "ivf.cuh"
#include "kmeans.cuh"
#include "prober.cuh"
#include "select.cuh"
#include "flat_scan.cuh"
#include "tc_ivf.cuh"
#include "tc_scan.cuh"
#include "timing.cuh"
#include "gemm_topk.cuh"
#include "topk.cuh"

namespace gn {

constexpr int TC_QCHUNK = 128;  // queries per tensor-core work unit (MMA N <= 128)

__device__ __forceinline__ int find_list_tc(const int64_t *item_off, int nc, int64_t item) {
    int lo = 0, hi = nc;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (item_off[mid] <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ void tc_units_body(int64_t i, const int64_t *__restrict__ item_off, int nc,
                              const int64_t *__restrict__ boff, const int64_t *__restrict__ list_off,
                              const int64_t *__restrict__ xoff, int rc, int qch, int64_t max_units,
                              TcUnit *__restrict__ units, int64_t *__restrict__ n_units) {
    const int64_t total = item_off[nc];
    if (i == 0) *n_units = min(total, max_units);
    if (i >= total || i >= max_units) return;
    const int l = find_list_tc(item_off, nc, i);
    const int64_t lb = list_off[l], le = list_off[l + 1];
    const int64_t nrc = (le - lb + rc - 1) / rc;
    const int64_t nqc = nrc > 0 ? (item_off[l + 1] - item_off[l]) / nrc : 1;
    const int64_t local = i - item_off[l];
    // the query chunks of one row chunk are adjacent: taken together by
    // different SMs, their second and later reads of the rows hit L2
    const int64_t rch = local / nqc, qc = local % nqc;
    TcUnit u;
    u.a0 = boff[l] + qc * qch;
    u.na = (int32_t)min((int64_t)qch, boff[l + 1] - u.a0);
    u.r0 = lb + rch * rc;
    u.r1 = min(le, u.r0 + rc);
    u.rbase = lb;
    u.xrow = xoff[l] + (u.r0 - lb);  // rc is a multiple of 128: stays tile-aligned
    units[i] = u;
}

// One launch for both: blocks [0, qb_blocks) fill Qb — row pos = the BF16 row
// of the query of the pair bucket[pos], with the pair's slot base and its
// query's score bound — the rest build the work units.  A warp moves QB_ROWS rows
// together: their loads (pair, then its query's row) are in flight at once, where
// one row a warp waited out each in turn (114,688 rows of 1 KB: 42 us,
// 27 here).
constexpr int QB_ROWS = 4;
__global__ void qb_units_kernel(const uint4 *__restrict__ q16, int K8, int np, const int64_t *__restrict__ bucket,
                                const int64_t *__restrict__ boff, int nc, const int64_t *__restrict__ qslot,
                                const int64_t *__restrict__ slot_rel, uint4 *__restrict__ qb,
                                int64_t *__restrict__ aslot, const uint32_t *__restrict__ qbound,
                                uint32_t *__restrict__ abound, int64_t max_pairs, unsigned qb_blocks,
                                const int64_t *__restrict__ item_off, const int64_t *__restrict__ list_off,
                                const int64_t *__restrict__ xoff, int rc, int qch, int64_t max_units,
                                TcUnit *__restrict__ units, int64_t *__restrict__ n_units) {
    if (blockIdx.x < qb_blocks) {
        const int lane = threadIdx.x & 31;
        const int64_t pos0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * QB_ROWS;
        const int64_t left = min(max_pairs, boff[nc]) - pos0;
        if (left <= 0) return;
        const int n = (int)min((int64_t)QB_ROWS, left);
        int64_t q = 0;
        if (lane < n) {
            const int64_t pair = bucket[pos0 + lane];
            q = pair / np;
            aslot[pos0 + lane] = qslot[q] + slot_rel[pair];
            abound[pos0 + lane] = qbound[q];
        }
        const uint4 *src[QB_ROWS];
#pragma unroll
        for (int r = 0; r < QB_ROWS; ++r) src[r] = q16 + __shfl_sync(0xffffffffu, q, r) * K8;
        uint4 *dst = qb + pos0 * K8;
#pragma unroll 2
        for (int j = lane; j < K8; j += 32) {
            uint4 v[QB_ROWS];
#pragma unroll
            for (int r = 0; r < QB_ROWS; ++r) v[r] = __ldg(src[r] + j);
#pragma unroll
            for (int r = 0; r < QB_ROWS; ++r)
                if (r < n) dst[(int64_t)r * K8 + j] = v[r];
        }
        return;
    }
    const int64_t i = (int64_t)(blockIdx.x - qb_blocks) * blockDim.x + threadIdx.x;
    tc_units_body(i, item_off, nc, boff, list_off, xoff, rc, qch, max_units, units, n_units);
}


// Two-sum of a and b: s = fl(a + b) and its exact rounding error.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float bp = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// Compensated accumulation of (a_i - b_i)^2 into (s, c): each square is split
// into its rounded product and the product's exact error (fma), the running
// sum keeps its rounding error (two-sum).
__device__ __forceinline__ void l2_acc4(const float4 a, const float4 b, int valid, float &s, float &c) {
    const float t[4] = {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z), __fsub_rn(a.w, b.w)};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (u < valid) {
            const float p = __fmul_rn(t[u], t[u]);
            const float e = __fmaf_rn(t[u], t[u], -p);
            float s2, err;
            two_sum(s, p, s2, err);
            s = s2;
            c = __fadd_rn(c, __fadd_rn(err, e));
        }
    }
}

// Combine the 32 lanes' (sum, error) pairs with two-sums; the result is
// within about one ulp of the exact sum.
__device__ __forceinline__ float l2_warp_total(float s, float c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float so = __shfl_xor_sync(0xffffffffu, s, o), co = __shfl_xor_sync(0xffffffffu, c, o);
        float s2, err;
        two_sum(s, so, s2, err);
        s = s2;
        c = __fadd_rn(c, __fadd_rn(co, err));
    }
    return __fadd_rn(s, c);
}

// Exact squared L2 (compensated FP32) of the query row q to the row x by one warp, for
// distances that l2sq_warp_pair cannot hold: it overflows only where the sum does.
__device__ __noinline__ float l2sq_warp_row(const float *__restrict__ q, const float *__restrict__ x, int d,
                                            int lane) {
    float s = 0.f, c = 0.f;
#pragma unroll 1
    for (int i = lane * 4; i < d; i += 128)
        l2_acc4(*reinterpret_cast<const float4 *>(q + i), __ldg(reinterpret_cast<const float4 *>(x + i)),
                min(4, d - i), s, c);
    return l2_warp_total(s, c);
}

// Exact squared L2 (compensated FP32) of the query row q to the rows x[0], x[1] by
// one warp, the first on lanes 0-15, the second on the others: lane l takes columns
// 4l..4l+3 of every 128-column block (coalesced float4 loads, all of a 512-column
// block issued together).  A sum that starts at the largest square of its lane is
// never below the square it takes next, so r = fl(s + t^2) is at most 2 s, s - r is
// exact, and fma(t, t, s - r) is the rounding error of r (to 2^-24 of itself): five
// packed steps for two squares, where the product's and the sum's errors taken
// separately (l2_acc4, no order assumed) need twelve for each.
__device__ __forceinline__ float l2sq_warp_pair(const float *__restrict__ q, const float *__restrict__ x0,
                                                const float *__restrict__ x1, int d, int lane) {
    const f32x2 minus = dup2(-1.f);
    float S[2] = {0.f, 0.f}, C[2] = {0.f, 0.f};
#pragma unroll 1
    for (int base = 0; base < d; base += 512) {
        f32x2 t[2][8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i0 = base + u * 128 + lane * 4;
            float4 qa = make_float4(0.f, 0.f, 0.f, 0.f), xa[2] = {qa, qa};
            if (base + u * 128 < d && i0 < d) {
                qa = __ldg(reinterpret_cast<const float4 *>(q + i0));
                xa[0] = __ldg(reinterpret_cast<const float4 *>(x0 + i0));
                xa[1] = __ldg(reinterpret_cast<const float4 *>(x1 + i0));
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                t[r][2 * u] = fma2(pack2(xa[r].x, xa[r].y), minus, pack2(qa.x, qa.y));
                t[r][2 * u + 1] = fma2(pack2(xa[r].z, xa[r].w), minus, pack2(qa.z, qa.w));
            }
        }
        if ((d & 3) && base + 512 >= d) {  // columns past d count nothing
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int valid = d - (base + u * 128 + lane * 4);
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float lo, hi;
                        unpack2(t[r][2 * u + h], lo, hi);
                        t[r][2 * u + h] = pack2(valid > 2 * h ? lo : 0.f, valid > 2 * h + 1 ? hi : 0.f);
                    }
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float m = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float lo, hi;
                unpack2(t[r][i], lo, hi);
                m = fmaxf(m, fmaxf(fabsf(lo), fabsf(hi)));
            }
            const float start = m * m;
            f32x2 s = dup2(start), c = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (base + u * 128 < d)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const f32x2 v = t[r][2 * u + h], sum = fma2(v, v, s);
                        c = add2(c, fma2(v, v, fma2(sum, minus, s)));
                        s = sum;
                    }
            float slo, shi, clo, chi, a, ea, b, eb, e;
            unpack2(s, slo, shi);
            unpack2(c, clo, chi);
            two_sum(slo, shi, a, ea);
            two_sum(a, -2.f * start, b, eb);
            two_sum(S[r], b, S[r], e);
            C[r] = __fadd_rn(C[r], __fadd_rn(__fadd_rn(clo, chi), __fadd_rn(__fadd_rn(ea, eb), e)));
        }
    }
    // the halves of the warp swap rows, then each adds up its own
    const bool up = lane & 16;
    float s = up ? S[1] : S[0], c = up ? C[1] : C[0];
    const float so = __shfl_xor_sync(0xffffffffu, up ? S[0] : S[1], 16),
                co = __shfl_xor_sync(0xffffffffu, up ? C[0] : C[1], 16);
    float s2, err;
    two_sum(s, so, s2, err);
    s = s2;
    c = __fadd_rn(c, __fadd_rn(co, err));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const float sx = __shfl_xor_sync(0xffffffffu, s, o), cx = __shfl_xor_sync(0xffffffffu, c, o);
        two_sum(s, sx, s2, err);
        s = s2;
        c = __fadd_rn(c, __fadd_rn(cx, err));
    }
    float out = __fadd_rn(s, c);
    if (__any_sync(0xffffffffu, !(out < INFINITY))) {  // the starts may overflow before the sums do
        const float a = l2sq_warp_row(q, x0, d, lane), b = l2sq_warp_row(q, x1, d, lane);
        out = up ? b : a;
    }
    return out;
}

// ── selection and exact re-rank ───────────────────────────────────────────
constexpr int SEL_P = 64;      // probes whose layout is held at a time (two per lane)
constexpr int SEL_GROUP = 128; // slots whose minima are held at a time (four per lane)
constexpr int SEL_BUF = 256;   // candidate keys per warp
constexpr int SEL_ALL = 512;   // candidate keys of a block's warps brought together
constexpr int SEL_WARPS = 28;  // warps resident per SM (72 registers a thread)

// Shared memory of one warp of the selection.
struct SelWarp {
    uint64_t buf[SEL_BUF];             // candidates (ordered score, row)
    uint64_t best[64];                 // the S best of them
    int4 probe[SEL_P];                 // list's first row, rows, first slot (from the query's), slots of the probes before
    uint16_t list[4 * SEL_GROUP];      // qualifying quarters: probe << 9 | quarter of the group
    int32_t pre[SEL_P + 1];            // slots of the probes before each
};

// A bound with at least S of the warp's values (R per lane) at or below it, and at
// most `more` others unless equal values leave no such bound: bit by bit from the
// highest in which the values differ.
template <int R>
__device__ __forceinline__ uint32_t warp_kth(const uint32_t (&v)[R], int S, int more) {
    uint32_t any = 0u, all = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        any |= v[i];
        all &= v[i];
    }
    any = __reduce_or_sync(0xffffffffu, any);
    all = __reduce_and_sync(0xffffffffu, all);
    if (any == all) return all;
    int bit = 31 - __clz((int)(any ^ all));
    uint32_t kth = bit == 31 ? 0u : all & ~((2u << bit) - 1u);
#pragma unroll 1
    for (; bit >= 0; --bit) {
        const uint32_t trial = kth | (1u << bit);
        int c = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) c += v[i] < trial;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c >= S && c <= S + more) return trial - 1u;
        if (c < S) kth = trial;
    }
    return kth;
}

// One group of slots of a query, slots g0 .. of the held probes (`all` of them): their
// quarter minima are read at once; `first` takes the threshold from them; the quarters
// at or below it are listed, and the listed quarters' scores read sixteen at a time,
// eight lanes to a quarter, their loads in flight together.  The first group is
// listed by every warp of the block, which read every NW-th sixteen of the list; a
// later one belongs to one warp.
template <int NW>
__device__ __forceinline__ void sel_group(SelWarp &W, const uint4 *__restrict__ tmin, const float *__restrict__ scores,
                                          int g0, int all, bool first, int S, int warp, int lane, uint32_t &tau,
                                          int &wn) {
    constexpr int U = SEL_GROUP / 32;
    const unsigned below = (1u << lane) - 1u;
    uint32_t v[4 * U];
    int probe[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int f = min(g0 + u * 32 + lane, all - 1);
        int p = 0;  // pre[p] <= f < pre[p + 1]
#pragma unroll
        for (int step = SEL_P / 2; step > 0; step >>= 1)
            if (W.pre[p + step] <= f) p += step;
        probe[u] = p;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int f = g0 + u * 32 + lane;
        uint4 m = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
        if (f < all) m = __ldg(tmin + W.probe[probe[u]].z + (f - W.probe[probe[u]].w));
        v[4 * u] = m.x;
        v[4 * u + 1] = m.y;
        v[4 * u + 2] = m.z;
        v[4 * u + 3] = m.w;
    }
    if (first && 4 * min(all - g0, SEL_GROUP) >= S) tau = min(tau, warp_kth<4 * U>(v, S, S / 8));
    int n = 0;  // listed
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const bool in = v[4 * u + e] <= tau;
            const unsigned b = __ballot_sync(0xffffffffu, in);
            if (in) W.list[n + __popc(b & below)] = (uint16_t)(probe[u] << 9 | (u * 32 + lane) * 4 + e);
            n += __popc(b);
        }
    __syncwarp();
#pragma unroll 1
    for (int e0 = first ? 16 * warp : 0; e0 < n; e0 += first ? 16 * NW : 16) {
        float4 x[4];
        uint32_t row[4];
        int rows[4];  // real rows among the lane's four
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = e0 + 4 * u + (lane >> 3);
            rows[u] = 0;
            if (i < n) {
                const int e = W.list[i];
                const int4 p = W.probe[e >> 9];
                const int s = g0 + (e >> 2 & (SEL_GROUP - 1)) - p.w, r = s * 128 + (e & 3) * 32 + (lane & 7) * 4;
                row[u] = (uint32_t)(p.x + r);
                rows[u] = p.y - r;
                if (rows[u] > 0)
                    x[u] = __ldg(reinterpret_cast<const float4 *>(scores + ((size_t)(p.z + s) * 128 + (r & 127))));
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (wn > SEL_BUF - 128) {  // the next four quarters may not fit
                tau = min(tau, list_cut<SEL_BUF / 32>(W.buf, wn, S));
                wn = S;
            }
            const float xs[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t bits = f2ord(xs[c]);
                const bool in = rows[u] > c && bits <= tau;
                const unsigned b = __ballot_sync(0xffffffffu, in);
                if (in) W.buf[wn + __popc(b & below)] = make_key(bits, row[u] + c);
                wn += __popc(b);
            }
        }
    }
    __syncwarp();
}

// Selection of one query by a block of NW warps.  The list scan leaves, per
// (query, list) pair, the scores of the list's rows in 128-row slots and the
// minimum score of every 32-row quarter of every slot.  Keys are (score, row),
// so ties go to the lower row.
//   threshold  tau = the S-th smallest quarter minimum of the query's first 128
//              slots, counted out of registers by every warp for itself: S
//              distinct rows score <= tau, so tau bounds the query's S-th best
//              score; capped by the query's bound from the probe stage, above
//              which the scan stored no quarter;
//   sweep      only the quarters with a minimum <= tau are read (a few dozen of
//              the query's hundreds); scores <= tau become keys in the warp's
//              buffer, cut to its best S when it fills, which lowers tau;
//   select     the S smallest keys of all the warps' buffers, by counting;
//   re-rank    two rows per warp at a time: exact squared L2 in FP32
//              (compensated sum); warp 0 returns the k nearest, ties to the
//              lower original index.
// Nothing but the hand-over of the candidates and of the distances (NW > 1) waits
// for another warp.  Measured on 400k x 512 rows, 1,024 lists, 28 probed, S 40: a batch
// of 4,096 took 203 us with block-wide radix selects, four warps a query (bound by their
// barriers, and by the twelve steps of each square), 78 us here, where its 336 MB of
// rows take 50 at the DRAM's measured rate; 16 queries (200k x 256, 16 of 512 lists)
// 35 us, split over 16 blocks each, 19 here.
template <int NW>
__global__ void __launch_bounds__(32 * NW, SEL_WARPS / NW) ivf_tc_select_kernel(
    const float *__restrict__ scores, const uint4 *__restrict__ tmin4, const uint32_t *__restrict__ qbound,
    const int32_t *__restrict__ probes, int np, const int64_t *__restrict__ qseg,
    const int64_t *__restrict__ seg_rel, const int64_t *__restrict__ list_off, int S, const float *__restrict__ Q,
    const float *__restrict__ X, int d, int dp, const int32_t *__restrict__ ids, int k,
    int64_t *__restrict__ out_idx, float *__restrict__ out_dist, int64_t *__restrict__ out_cnt, const int *err,
    int *status) {
    __shared__ SelWarp s_warp[NW];
    if (status && blockIdx.x == 0 && threadIdx.x == 0) *status = *err;
    __shared__ uint64_t s_all[NW > 1 ? SEL_ALL : 1];
    __shared__ int s_wn[NW];
    __shared__ float s_d[64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t q = blockIdx.x;
    SelWarp &W = s_warp[warp];
    const uint4 *tmin = tmin4 + qseg[q];
    const float *sc = scores + qseg[q] * 128;
    uint32_t tau = qbound[q];  // scores <= tau are candidates
    int wn = 0;                // keys in this warp's buffer
    int group = 0;
    for (int p0 = 0; p0 < np; p0 += SEL_P) {
        // the probes' layout: lane l holds probes l and l + 32
        int ns[2];
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = h * 32 + lane;
            const int32_t l = p0 + i < np ? probes[q * np + p0 + i] : -1;
            int64_t lb = 0, len = 0, sl = 0;
            if (l >= 0) {
                lb = list_off[l];
                len = list_off[l + 1] - lb;
                sl = seg_rel[q * np + p0 + i];
            }
            W.probe[i] = make_int4((int)lb, (int)len, (int)sl, 0);
            ns[h] = (int)((len + 127) >> 7);
        }
        int inc0 = ns[0], inc1 = ns[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, inc0, o), b = __shfl_up_sync(0xffffffffu, inc1, o);
            if (lane >= o) {
                inc0 += a;
                inc1 += b;
            }
        }
        inc1 += __shfl_sync(0xffffffffu, inc0, 31);
        W.pre[lane + 1] = inc0;
        W.pre[lane + 33] = inc1;
        W.probe[lane].w = inc0 - ns[0];
        W.probe[lane + 32].w = inc1 - ns[1];
        if (lane == 0) W.pre[0] = 0;
        __syncwarp();
        const int all = W.pre[SEL_P];
        for (int g0 = 0; g0 < all; g0 += SEL_GROUP, ++group)
            if (group == 0 || NW == 1 || group % NW == warp)
                sel_group<NW>(W, tmin, sc, g0, all, group == 0, S, warp, lane, tau, wn);
    }
    __syncwarp();
    int m;  // candidates re-ranked: best[0 .. m)
    if (NW == 1) {
        m = warp_best(W.buf, wn, S, W.best);
    } else {  // brought together, then every warp selects for itself
        if (lane == 0) s_wn[warp] = wn;
        __syncthreads();
        int total = 0, before = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            if (w == warp) before = total;
            total += s_wn[w];
        }
        if (total <= SEL_ALL) {
            for (int i = lane; i < wn; i += 32) s_all[before + i] = W.buf[i];
            __syncthreads();
            m = warp_best(s_all, total, S, W.best);
        } else {
            m = warp_best_of(
                [&](int i) {
                    int w = 0;
                    while (i >= s_wn[w]) i -= s_wn[w++];
                    return s_warp[w].buf[i];
                },
                total, S, W.best);
        }
    }
    __syncwarp();
    // exact re-rank, two rows per warp at a time.  A warp of a small batch asks for all
    // its rows first, so that they come in one DRAM round trip; a large batch has
    // enough other warps to cover that wait.
    const float *qrow = Q + q * dp;
    if (NW > 1) {
        const int lines = (d * 4 + 127) / 128;
        for (int r = 2 * warp; r < m; r += 2 * NW)
            for (int i = lane; i < 2 * lines; i += 32) {
                const int u = i >= lines;
                if (r + u < m)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(X + (int64_t)key_idx(W.best[r + u]) * dp +
                                                                  (i - u * lines) * 32));
            }
    }
    uint32_t id[2] = {0u, 0u};
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (warp == 0 && h * 32 + lane < m) id[h] = (uint32_t)ids[key_idx(W.best[h * 32 + lane])];
#pragma unroll 1
    for (int r = 2 * warp; r < m; r += 2 * NW) {
        const bool two = r + 1 < m;
        const float *x0 = X + (int64_t)key_idx(W.best[r]) * dp;
        const float dist = l2sq_warp_pair(qrow, x0, two ? X + (int64_t)key_idx(W.best[r + 1]) * dp : x0, d, lane);
        if (lane == 0 || (lane == 16 && two)) s_d[r + (lane >> 4)] = dist;
    }
    if (NW > 1) __syncthreads();
    else __syncwarp();
    if (warp != 0) return;
    uint64_t key[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        key[h] = h * 32 + lane < m ? make_key(__float_as_uint(s_d[h * 32 + lane]), id[h]) : KEY_EMPTY;
    warp_sort<2>(key);
    const bool e = key[0] == KEY_EMPTY;
    if (lane < k) {
        out_idx[q * k + lane] = e ? -1 : (int64_t)key_idx(key[0]);
        out_dist[q * k + lane] = e ? 0.f : __uint_as_float(key_dist(key[0]));
    }
    const int cnt = __popc(__ballot_sync(0xffffffffu, lane < k && !e));
    if (lane == 0 && out_cnt) out_cnt[q] = cnt;
}

// Warps per query (8, 4, 2 or 1) of the kernels that give a query a block: the most
// that fit the GPU at once, SEL_WARPS per SM, so that a small batch has its query's work
// split and a large one has no more warps than can be resident.
template <typename Launch>
static void warps_per_query(int64_t nq, int fixed, Launch &&launch) {
    int nw = 8;
    while (nw > 1 && nq * nw > (int64_t)dev_info().num_sms * SEL_WARPS) nw /= 2;
    if (fixed) nw = fixed;
    if (nw == 8) launch(std::integral_constant<int, 8>());
    else if (nw == 4) launch(std::integral_constant<int, 4>());
    else if (nw == 2) launch(std::integral_constant<int, 2>());
    else launch(std::integral_constant<int, 1>());
}

// ── tensor-core coarse stage ──────────────────────────────────────────────
// Units of the centroid scan: every query chunk of 256 against every chunk of
// 128 centroids; aslot[q] = q * nc so the scores land row-major [nq x nc].
__global__ void coarse_units_kernel(int64_t nq, int nc, TcUnit *__restrict__ units, int64_t *__restrict__ n_units,
                                    int64_t *__restrict__ aslot) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nqc = (nq + TC_QCHUNK - 1) / TC_QCHUNK, ncc = (nc + 127) / 128;
    if (t == 0) *n_units = nqc * ncc;
    if (t < nq) aslot[t] = t * nc;
    if (t >= nqc * ncc) return;
    const int64_t qc = t / ncc, cc = t % ncc;
    TcUnit u;
    u.a0 = qc * TC_QCHUNK;
    u.na = (int32_t)min((int64_t)TC_QCHUNK, nq - u.a0);
    u.r0 = cc * 128;
    u.r1 = min((int64_t)nc, u.r0 + 128);
    u.rbase = 0;
    u.xrow = u.r0;
    units[t] = u;
}

constexpr int PROBE_MAX_D = 2048;

// The query's score bound for the list scan, from b = this thread's probed
// candidate list's distance bound (+inf for threads without one): with D the
// smallest b, at least `shortlist` scored rows x have |q - x|^2 <= D, so the
// shortlist-th smallest exact score |x|^2 - 2 q.x is at most D - |q|^2.  The
// scan's BF16 score differs from the exact one by at most
// 2 |q.x - acc| + rounding <= 2 (2^-7 + 2^-16 + 2^-9 (1 + 2^-8)^2) |q| |x| + ...
// (both operands rounded to 8 significant bits; 2^-9 of sum |q_i x_i| allowed
// for the tensor core's accumulation, far above FP32's), so the bound adds
// 0.03 |q| xmax + 2^-12 (xmax + |q|)^2 and rounds every other term outwards.
// All ones when there is none.
__device__ __forceinline__ uint32_t probe_bound_key(float D, float qn, float xmax) {
    const float qa = sqrtf(qn);
    const float B = D * (1.f + 1.f / 1024.f) - qn * (1.f - 1.f / 1024.f) + 0.03f * qa * xmax +
                    (xmax + qa) * (xmax + qa) * (1.f / 4096.f);
    return (B < INFINITY && B == B) ? f2ord(B) : 0xffffffffu;
}

// |q|^2 by one warp
__device__ __forceinline__ float warp_sqnorm(const float *__restrict__ q, int d, int lane) {
    float s = 0.f;
    for (int t = lane; t < d; t += 32) s = fmaf(q[t], q[t], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// The PROBER_CAND smallest keys (score, centroid) of a query's nc >= PROBER_CAND scores
// into best, by one warp: a threshold out of 32 R group minima held in registers
// (every 32 R-th score a group), then the best of the scores at or below it.
template <int R>
__device__ __forceinline__ void probe_candidates(const float *__restrict__ sq, int nc, uint64_t *buf, uint64_t *best,
                                                 int lane) {
    constexpr int NC = PROBER_CAND;
    uint32_t v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        v[i] = 0xffffffffu;
        if (i * 32 < nc && i * 32 + lane < nc) v[i] = f2ord(__ldg(sq + i * 32 + lane));
    }
#pragma unroll 1
    for (int g = 32 * R; g < nc; g += 32 * R)
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (g + i * 32 + lane < nc) v[i] = min(v[i], f2ord(__ldg(sq + g + i * 32 + lane)));
    uint32_t tau = warp_kth<R>(v, NC, NC / 2);
    int wn = 0;
#pragma unroll 1
    for (int g = 0; g < nc; g += 32 * R)
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int c = g + i * 32 + lane;
            if (g + i * 32 >= nc) break;
            const uint32_t bits = nc <= 32 * R ? v[i] : c < nc ? f2ord(__ldg(sq + c)) : 0xffffffffu;
            const bool in = c < nc && bits <= tau;
            const unsigned b = __ballot_sync(0xffffffffu, in);
            if (b == 0) continue;
            if (in) buf[wn + __popc(b & ((1u << lane) - 1u))] = make_key(bits, (uint32_t)c);
            wn += __popc(b);
            if (wn > SEL_BUF - 32) {
                tau = min(tau, list_cut<SEL_BUF / 32>(buf, wn, NC));
                wn = NC;
            }
        }
    __syncwarp();
    const int ntop = warp_best(buf, wn, NC, best);
    for (int i = ntop + lane; i < NC; i += 32) best[i] = KEY_EMPTY;
    __syncwarp();
}

// Per query (block of NW warps): the 64 best centroids by BF16 score, their
// exact squared distances (FP32), sorted nearest first; then the first np of them
// (PROBE_FIXED), the learned prober's choice (PROBE_MLP, fused here) or, for
// mlp_probe_kernel, all of them with their features (PROBE_CANDS).
// The candidates are the 64 smallest keys (BF16 score, centroid), counted by one
// warp; the distances are split over the warps, four candidates at a time.  Measured with
// 1,024 centroids of 512 dimensions: 88 us for 4,096 queries with a block-wide radix
// select, 49 here (their 537 MB of centroid rows come from L2).
enum { PROBE_FIXED, PROBE_MLP, PROBE_CANDS };
template <int MODE, int NW>
__global__ void __launch_bounds__(32 * NW, SEL_WARPS / NW)
    coarse_probe_kernel(const float *__restrict__ scores, int nc, const float *__restrict__ Q, int d, int dp,
                        const float *__restrict__ C, int np, ProberWeights w, float logit_tau,
                        int32_t *__restrict__ probes, int32_t *__restrict__ nprobed,
                        const float *__restrict__ rho, int shortlist, float xmax,
                        uint32_t *__restrict__ qbound, float *__restrict__ feat_out, int32_t *__restrict__ cand_out,
                        float *__restrict__ cb_out, float *__restrict__ qn_out) {
    constexpr int NC = PROBER_CAND, H = PROBER_HIDDEN;
    constexpr bool MLP = MODE == PROBE_MLP;
    static_assert(H == 256 && NC == 64, "warp-per-row MLP layout: 32 lanes x 8 weights, 8 warps x 8 candidates");
    static_assert(!MLP || NW == 8, "one thread per hidden unit");
    __shared__ uint64_t buf[SEL_BUF], best[NC];
    __shared__ float sd[NC];
    const int64_t q = blockIdx.x;
    const int j = threadIdx.x, lane = j & 31, warp = j >> 5;
    const float *sq = scores + q * nc, *qrow = Q + q * dp;
    if (warp == 0) {
        if (nc <= 512) probe_candidates<16>(sq, nc, buf, best, lane);
        else probe_candidates<32>(sq, nc, buf, best, lane);
    }
    if (NW > 1) __syncthreads();
    {   // exact squared distances, four candidates together: each load instruction
        // reads 512 contiguous bytes of a centroid row
        const float4 *qr = reinterpret_cast<const float4 *>(qrow);
        const int n4 = d >> 2;
#pragma unroll 1
        for (int i0 = 4 * warp; i0 < NC; i0 += 4 * NW) {
            const float *cr[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint64_t key = best[i0 + u];
                cr[u] = C + (int64_t)(key == KEY_EMPTY ? 0 : key_idx(key)) * dp;
            }
            float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
            for (int t = lane; t < n4; t += 32) {
                const float4 b = __ldg(qr + t);
                float4 a[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) a[u] = __ldg(reinterpret_cast<const float4 *>(cr[u]) + t);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float e0 = b.x - a[u].x, e1 = b.y - a[u].y, e2 = b.z - a[u].z, e3 = b.w - a[u].w;
                    s0[u] = fmaf(e0, e0, s0[u]);
                    s1[u] = fmaf(e1, e1, s1[u]);
                    s0[u] = fmaf(e2, e2, s0[u]);
                    s1[u] = fmaf(e3, e3, s1[u]);
                }
            }
            for (int t = (n4 << 2) + lane; t < d; t += 32)  // d % 4 tail
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float e = qrow[t] - cr[u][t];
                    s0[u] = fmaf(e, e, s0[u]);
                }
            // the four sums over the lanes: lanes 0, 8, 16, 24 end with candidates 0, 2, 1, 3's
            const bool h16 = lane & 16, h8 = lane & 8;
            float x = s0[0] + s1[0], y = s0[1] + s1[1];
            float p = (h16 ? y : x) + __shfl_xor_sync(0xffffffffu, h16 ? x : y, 16);
            x = s0[2] + s1[2];
            y = s0[3] + s1[3];
            const float p2 = (h16 ? y : x) + __shfl_xor_sync(0xffffffffu, h16 ? x : y, 16);
            p = (h8 ? p2 : p) + __shfl_xor_sync(0xffffffffu, h8 ? p : p2, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
            if ((lane & 7) == 0) sd[i0 + (h8 ? 2 : 0) + (h16 ? 1 : 0)] = p;
        }
    }
    __shared__ float s_qn;
    if (warp == NW - 1 && !MLP && qbound) {
        const float qn = warp_sqnorm(qrow, d, lane);
        if (lane == 0) s_qn = qn;
    }
    if (NW > 1) __syncthreads();
    else __syncwarp();
    __shared__ int32_t sc[MLP ? NC : 1];
    __shared__ float sf[MLP ? NC : 1], sb[MLP ? NC : 1];
    if (warp == 0) {
        uint64_t key[2];  // sorted: lane l holds positions l and l + 32
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = h * 32 + lane;
            const uint64_t c = best[i];
            key[h] = c == KEY_EMPTY ? KEY_EMPTY : make_key(__float_as_uint(sd[i]), key_idx(c));
        }
        warp_sort<2>(key);
        const float d1 = __shfl_sync(0xffffffffu, __uint_as_float(key_dist(key[0])), 0);
        float near = INFINITY;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = h * 32 + lane;
            const bool e = key[h] == KEY_EMPTY;
            const int32_t c = e ? -1 : (int32_t)key_idx(key[h]);
            // bound on the squared distance of the query's shortlist-th nearest row if
            // this list is probed: its `shortlist` rows nearest the centroid lie within
            // rho of it, hence within |q - c| + rho of the query
            float b = INFINITY;
            if (qbound && !e) {
                const float r = rho[(size_t)c * IVF_RHO + shortlist - 1];
                if (r < INFINITY) {
                    const float t = sqrtf(__uint_as_float(key_dist(key[h])) * (1.f + 1.f / 1024.f)) + r;
                    b = t * t;
                }
            }
            const float f =
                e ? 0.f : fmaxf(0.f, 1.f - (__uint_as_float(key_dist(key[h])) - d1) / fmaxf(d1, 1e-12f));
            if (MLP) {
                sc[i] = c;
                sf[i] = f;
                sb[i] = b;
            } else if (MODE == PROBE_CANDS) {
                cand_out[q * NC + i] = c;
                feat_out[q * NC + i] = f;
                cb_out[q * NC + i] = b;
            } else if (i < np) {
                probes[q * np + i] = c;
                near = fminf(near, b);
            }
        }
        if (MODE == PROBE_CANDS && lane == 0) qn_out[q] = s_qn;
        if (MODE == PROBE_FIXED && qbound) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) near = fminf(near, __shfl_xor_sync(0xffffffffu, near, o));
            if (lane == 0) qbound[q] = probe_bound_key(near, s_qn, xmax);
        }
    }
    if (!MLP) return;
    __shared__ float sz[MLP ? NC : 1], sred[4];
    __shared__ __align__(16) float sh1[MLP ? H : 4], sh2[MLP ? H : 4];
    __shared__ int s_cnt0;
    __syncthreads();
    const __nv_bfloat16 *W1 = reinterpret_cast<const __nv_bfloat16 *>(w.W1);
    const __nv_bfloat16 *W2 = reinterpret_cast<const __nv_bfloat16 *>(w.W2);
    const __nv_bfloat16 *W3 = reinterpret_cast<const __nv_bfloat16 *>(w.W3);
    // layer 1: thread j = hidden unit j, gathered rows of W1 (loads issued ahead)
    float a = w.b1[j];
#pragma unroll 32
    for (int i = 0; i < NC; ++i) {
        const int c = sc[i];
        const float wv = c >= 0 ? __bfloat162float(W1[(size_t)c * H + j]) : 0.f;
        a = fmaf(sf[i], wv, a);
    }
    sh1[j] = fmaxf(a, 0.f);
    __syncthreads();
    // layer 2: warp w computes outputs 32w .. 32w + 31, one W2 row (512 bytes,
    // lane l its 16 bytes) per load instruction, four rows in flight; lane l
    // holds h1[8l .. 8l + 7]
    {
        const float4 *h4 = reinterpret_cast<const float4 *>(sh1);
        const float4 x0 = h4[2 * lane], x1 = h4[2 * lane + 1];
        const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll 1
        for (int r0 = warp * 32; r0 < warp * 32 + 32; r0 += 4) {
            uint4 u[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) u[k] = __ldg(reinterpret_cast<const uint4 *>(W2 + (size_t)(r0 + k) * H) + lane);
            float acc[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u[k]);
                float t = 0.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(h[e]);
                    t = fmaf(f.x, xs[2 * e], t);
                    t = fmaf(f.y, xs[2 * e + 1], t);
                }
                acc[k] = t;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (lane == k) sh2[r0 + k] = fmaxf(acc[k] + w.b2[r0 + k], 0.f);
        }
    }
    __syncthreads();
    // layer 3: one warp per candidate (eight per warp, four in flight), its W3
    // row in one load instruction
    {
        const float4 *h4 = reinterpret_cast<const float4 *>(sh2);
        const float4 x0 = h4[2 * lane], x1 = h4[2 * lane + 1];
        const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll 1
        for (int k0 = 0; k0 < 8; k0 += 4) {
            uint4 u[4];
            int cs[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                cs[k] = sc[warp + 8 * (k0 + k)];
                u[k] = cs[k] >= 0 ? __ldg(reinterpret_cast<const uint4 *>(W3 + (size_t)cs[k] * H) + lane)
                                  : make_uint4(0u, 0u, 0u, 0u);
            }
            float acc[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u[k]);
                float t = 0.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(h[e]);
                    t = fmaf(f.x, xs[2 * e], t);
                    t = fmaf(f.y, xs[2 * e + 1], t);
                }
                acc[k] = t;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < 4; ++k) sz[warp + 8 * (k0 + k)] = cs[k] >= 0 ? acc[k] + w.b3[cs[k]] : -INFINITY;
        }
    }
    __syncthreads();
    bool keep = false;
    unsigned m = 0;
    const int i = warp * 32 + lane;
    if (warp < NC / 32) {
        keep = sc[i] >= 0 && (i == 0 || sz[i] >= logit_tau);
        m = __ballot_sync(0xffffffffu, keep);
        if (warp == 0 && lane == 0) s_cnt0 = __popc(m);
    }
    __syncthreads();
    if (warp < NC / 32) {
        const int pos = (warp == 0 ? 0 : s_cnt0) + __popc(m & ((1u << lane) - 1u));
        if (keep) probes[q * NC + pos] = sc[i];
        if (warp == 1) {
            const int total = s_cnt0 + __popc(m);
            for (int t = total + lane; t < NC; t += 32) probes[q * NC + t] = -1;
            if (lane == 0 && nprobed) nprobed[q] = total;
        }
    }
    if (qbound) {
        float b = keep ? sb[i] : INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b = fminf(b, __shfl_xor_sync(0xffffffffu, b, o));
        if (lane == 0 && warp < 2) sred[warp] = b;
        if (warp == 2) {
            const float qs = warp_sqnorm(qrow, d, lane);
            if (lane == 0) sred[2] = qs;
        }
        __syncthreads();
        if (j == 0) qbound[q] = probe_bound_key(fminf(sred[0], sred[1]), sred[2], xmax);
    }
}

// The prober and its probe choice for MLP_QB queries per block (large batches, from
// coarse_probe_kernel<PROBE_CANDS>'s candidates and features):
//   layer 1  thread j = hidden unit j: the candidates' rows of W1, gathered,
//            query by query, 32 loads in flight;
//   layer 2  thread j = hidden unit j for the block's queries, its W2 row
//            read once (16-byte loads), the queries' first-layer outputs from
//            shared memory;
//   layer 3  warp w = query w: its 64 candidate lists' W3 rows (one 512-byte
//            row per load instruction, four in flight) against the query's
//            second-layer output;
//   choice   the nearest candidate always, the others whose logit is at
//            least the threshold, in distance order; the list scan's score
//            bound from the chosen lists.
// The arithmetic (FP32 accumulation of BF16 weights, same order per dot
// product within a lane) matches the fused kernel's up to summation order.
constexpr int MLP_QB = 8;
constexpr int64_t MLP_BATCH_MIN = 1024;  // smaller batches keep the MLP fused in coarse_probe_kernel
__global__ void __launch_bounds__(256) mlp_probe_kernel(const float *__restrict__ feat,
                                                        const int32_t *__restrict__ cand,
                                                        const float *__restrict__ cb, const float *__restrict__ qnv,
                                                        int64_t nq, ProberWeights w, float logit_tau, float xmax,
                                                        int32_t *__restrict__ probes, int32_t *__restrict__ nprobed,
                                                        uint32_t *__restrict__ qbound) {
    constexpr int NC = PROBER_CAND, H = PROBER_HIDDEN;
    __shared__ __align__(16) float h1s[MLP_QB][H], h2s[MLP_QB][H];
    const int j = threadIdx.x, lane = j & 31, warp = j >> 5;
    const int64_t q0 = (int64_t)blockIdx.x * MLP_QB;
    const int nqb = (int)min((int64_t)MLP_QB, nq - q0);
    __shared__ int32_t s_c[MLP_QB][NC];
    __shared__ float s_f[MLP_QB][NC];
    for (int i = j; i < MLP_QB * NC; i += 256) {
        const bool in = i / NC < nqb;
        s_c[i / NC][i % NC] = in ? cand[q0 * NC + i] : -1;
        s_f[i / NC][i % NC] = in ? feat[q0 * NC + i] : 0.f;
    }
    __syncthreads();
    {   // layer 1
        const __nv_bfloat16 *W1 = reinterpret_cast<const __nv_bfloat16 *>(w.W1);
        const float b1 = w.b1[j];
#pragma unroll 1
        for (int qq = 0; qq < MLP_QB; ++qq) {
            float a = b1;
#pragma unroll 32
            for (int i = 0; i < NC; ++i) {
                const int c = s_c[qq][i];
                const float wv = c >= 0 ? __bfloat162float(W1[(size_t)c * H + j]) : 0.f;
                a = fmaf(s_f[qq][i], wv, a);
            }
            h1s[qq][j] = fmaxf(a, 0.f);
        }
    }
    __syncthreads();
    {   // layer 2
        const __nv_bfloat16 *W2 = reinterpret_cast<const __nv_bfloat16 *>(w.W2);
        const uint4 *row = reinterpret_cast<const uint4 *>(W2 + (size_t)j * H);
        float acc[MLP_QB];
#pragma unroll
        for (int qq = 0; qq < MLP_QB; ++qq) acc[qq] = 0.f;
#pragma unroll 4
        for (int i8 = 0; i8 < H / 8; ++i8) {
            const uint4 u = __ldg(row + i8);
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
            float wv[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h[e]);
                wv[2 * e] = f.x;
                wv[2 * e + 1] = f.y;
            }
#pragma unroll
            for (int qq = 0; qq < MLP_QB; ++qq) {
                const float4 x0 = *reinterpret_cast<const float4 *>(&h1s[qq][8 * i8]);
                const float4 x1 = *reinterpret_cast<const float4 *>(&h1s[qq][8 * i8 + 4]);
                acc[qq] = fmaf(wv[0], x0.x, acc[qq]);
                acc[qq] = fmaf(wv[1], x0.y, acc[qq]);
                acc[qq] = fmaf(wv[2], x0.z, acc[qq]);
                acc[qq] = fmaf(wv[3], x0.w, acc[qq]);
                acc[qq] = fmaf(wv[4], x1.x, acc[qq]);
                acc[qq] = fmaf(wv[5], x1.y, acc[qq]);
                acc[qq] = fmaf(wv[6], x1.z, acc[qq]);
                acc[qq] = fmaf(wv[7], x1.w, acc[qq]);
            }
        }
        const float b2 = w.b2[j];
#pragma unroll
        for (int qq = 0; qq < MLP_QB; ++qq) h2s[qq][j] = fmaxf(acc[qq] + b2, 0.f);
    }
    __syncthreads();
    if (warp >= nqb) return;
    const int64_t q = q0 + warp;
    // layer 3 for this warp's query: lane l holds h2[8l .. 8l + 7]
    const __nv_bfloat16 *W3 = reinterpret_cast<const __nv_bfloat16 *>(w.W3);
    const float4 x0 = *reinterpret_cast<const float4 *>(&h2s[warp][8 * lane]);
    const float4 x1 = *reinterpret_cast<const float4 *>(&h2s[warp][8 * lane + 4]);
    const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    const int32_t c_lo = cand[q * NC + lane], c_hi = cand[q * NC + 32 + lane];
    float z_lo = -INFINITY, z_hi = -INFINITY;
#pragma unroll 1
    for (int i0 = 0; i0 < NC; i0 += 4) {
        uint4 u[4];
        int cs[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            cs[k] = __shfl_sync(0xffffffffu, (i0 + k) < 32 ? c_lo : c_hi, (i0 + k) & 31);
            u[k] = cs[k] >= 0 ? __ldg(reinterpret_cast<const uint4 *>(W3 + (size_t)cs[k] * H) + lane)
                              : make_uint4(0u, 0u, 0u, 0u);
        }
        float acc[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u[k]);
            float t = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h[e]);
                t = fmaf(f.x, xs[2 * e], t);
                t = fmaf(f.y, xs[2 * e + 1], t);
            }
            acc[k] = t;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + k;
            const float z = cs[k] >= 0 ? acc[k] + w.b3[cs[k]] : -INFINITY;
            if (i < 32 && lane == i) z_lo = z;
            if (i >= 32 && lane == i - 32) z_hi = z;
        }
    }
    // the choice: candidate 0 always, the others at or above the threshold
    const bool k_lo = c_lo >= 0 && (lane == 0 || z_lo >= logit_tau);
    const bool k_hi = c_hi >= 0 && z_hi >= logit_tau;
    const unsigned m_lo = __ballot_sync(0xffffffffu, k_lo), m_hi = __ballot_sync(0xffffffffu, k_hi);
    const int n_lo = __popc(m_lo);
    if (k_lo) probes[q * NC + __popc(m_lo & ((1u << lane) - 1u))] = c_lo;
    if (k_hi) probes[q * NC + n_lo + __popc(m_hi & ((1u << lane) - 1u))] = c_hi;
    const int total = n_lo + __popc(m_hi);
    for (int t = total + lane; t < NC; t += 32) probes[q * NC + t] = -1;
    if (lane == 0 && nprobed) nprobed[q] = total;
    if (qbound) {
        float b = fminf(k_lo ? cb[q * NC + lane] : INFINITY, k_hi ? cb[q * NC + 32 + lane] : INFINITY);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b = fminf(b, __shfl_xor_sync(0xffffffffu, b, o));
        if (lane == 0) qbound[q] = probe_bound_key(b, qnv[q], xmax);
    }
}

// Probes of the tensor-core engine: BF16 centroid scores on the tensor cores,
// exact re-rank of the 64 best, then fixed n_probe or the learned prober.
static int ivfl2_probes_tc(gn_index *ix, const float *dQ, int64_t nq, int *np_out, cudaStream_t st) {
    IvfL2State &S = *ix->ivfl2;
    IvfScratch &T = S.s;
    // per query: the list scan's score bound (all ones: none, every score kept)
    GN_TRY(T.qbound.ensure((size_t)std::max<int64_t>(nq, 1) * 4));
    if (S.nc < PROBER_CAND || S.d > PROBE_MAX_D || S.nc > 8192) {  // outside the 64-candidate stage's limits
        if (S.prober) return fail(GN_ERR_INVALID, "learned probing needs at least 64 lists");
        int np = std::min<int32_t>(S.nprobe, S.nc);
        *np_out = np;
        GN_CUDA_TRY(cudaMemsetAsync(T.qbound.p, 0xff, (size_t)nq * 4, st));
        return ivfl2_coarse(ix, dQ, nq, np, st);
    }
    const bool mlp = S.prober != nullptr;
    const int np = mlp ? PROBER_CAND : std::min<int32_t>(std::min<int32_t>(S.nprobe, S.nc), PROBER_CAND);
    if (!mlp && S.nprobe > PROBER_CAND) {  // wider fixed probing: the FP32 coarse stage
        *np_out = std::min<int32_t>(S.nprobe, S.nc);
        GN_CUDA_TRY(cudaMemsetAsync(T.qbound.p, 0xff, (size_t)nq * 4, st));
        return ivfl2_coarse(ix, dQ, nq, *np_out, st);
    }
    *np_out = np;
    const int64_t units = ceil_div(nq, TC_QCHUNK) * ceil_div(S.nc, 128);
    GN_TRY(S.cunits.ensure((size_t)units * sizeof(TcUnit)));
    GN_TRY(S.cnunits.ensure(8));
    GN_TRY(S.caslot.ensure((size_t)nq * 8));
    GN_TRY(S.cscores.ensure((size_t)nq * S.nc * 4));
    GN_TRY(T.probes.ensure((size_t)nq * np * 4));
    coarse_units_kernel<<<(unsigned)ceil_div(std::max<int64_t>(units, nq), 256), 256, 0, st>>>(
        nq, S.nc, S.cunits.as<TcUnit>(), S.cnunits.as<int64_t>(), S.caslot.as<int64_t>());
    TcIvfLaunch a;
    a.X = S.c16.p;
    a.x_rows = std::max<int64_t>(S.nc, 128);
    a.Q = S.q16.p;
    a.q_rows = std::max<int64_t>(nq, 256);
    a.K = S.K;
    a.units = S.cunits.as<TcUnit>();
    a.n_units = S.cnunits.as<int64_t>();
    a.xnorm = S.cnorm.as<float>();
    a.aslot = S.caslot.as<int64_t>();
    a.scores = S.cscores.as<float>();
    a.err = S.err.as<int>();
    a.next_unit = S.sched.as<unsigned long long>() + 0;
    a.grid = (int)std::min<int64_t>(dev_info().num_sms, units);
    GN_TRY(tc_ivf_launch(a, st));
    ProberWeights w;
    float *feat = nullptr, *cbnd = nullptr, *qnv = nullptr;
    int32_t *cand = nullptr;
    if (mlp) {
        GN_TRY(prober_weights(S.prober, &w));
        GN_TRY(T.nprobed.ensure((size_t)nq * 4));
        if (nq >= MLP_BATCH_MIN) {  // the MLP batched over 8 queries per block
            GN_TRY(T.mfeat.ensure((size_t)nq * PROBER_CAND * 4));
            GN_TRY(T.mcand.ensure((size_t)nq * PROBER_CAND * 4));
            GN_TRY(T.mcb.ensure((size_t)nq * PROBER_CAND * 4));
            GN_TRY(T.mqn.ensure((size_t)nq * 4));
            feat = T.mfeat.as<float>();
            cand = T.mcand.as<int32_t>();
            cbnd = T.mcb.as<float>();
            qnv = T.mqn.as<float>();
        }
        auto probe = [&](auto MODEC, auto NWC) {
            constexpr int MODE = decltype(MODEC)::value, NW = decltype(NWC)::value;
            coarse_probe_kernel<MODE, NW><<<(unsigned)nq, 32 * NW, 0, st>>>(
                S.cscores.as<float>(), S.nc, dQ, S.d, S.dp, S.cent.as<float>(), np, w, S.prober_tau,
                T.probes.as<int32_t>(), T.nprobed.as<int32_t>(), S.rho.as<float>(), S.shortlist, S.xmax,
                T.qbound.as<uint32_t>(), feat, cand, cbnd, qnv);
        };
        if (feat) {
            warps_per_query(nq, 0, [&](auto NWC) { probe(std::integral_constant<int, PROBE_CANDS>(), NWC); });
            mlp_probe_kernel<<<(unsigned)ceil_div(nq, MLP_QB), 256, 0, st>>>(
                feat, cand, cbnd, qnv, nq, w, S.prober_tau, S.xmax, T.probes.as<int32_t>(),
                T.nprobed.as<int32_t>(), T.qbound.as<uint32_t>());
        } else {
            probe(std::integral_constant<int, PROBE_MLP>(), std::integral_constant<int, 8>());
        }
    } else {
        warps_per_query(nq, 0, [&](auto NWC) {
            constexpr int NW = decltype(NWC)::value;
            coarse_probe_kernel<PROBE_FIXED, NW><<<(unsigned)nq, 32 * NW, 0, st>>>(
                S.cscores.as<float>(), S.nc, dQ, S.d, S.dp, S.cent.as<float>(), np, w, 0.f, T.probes.as<int32_t>(),
                nullptr, S.rho.as<float>(), S.shortlist, S.xmax, T.qbound.as<uint32_t>(), nullptr, nullptr, nullptr,
                nullptr);
        });
    }
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

// FP32 list rows (dp floats) -> the tiled BF16 layout of IvfL2State::x16:
// thread per (row, 8 values); row r of list l goes to padded row
// p = xoff[l] + (r - list_off[l]), tile p / 128, and its K slice kb to the
// 16 KB block (tile * K/64 + kb); values past d are zero.
__global__ void x16_tiled_kernel(const float *__restrict__ X, int64_t n, int d, int dp,
                                 const int64_t *__restrict__ list_off, int nc, const int64_t *__restrict__ xoff,
                                 int K, uint4 *__restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int g8 = K / 8;
    const int64_t r = t / g8;
    if (r >= n) return;
    const int g = (int)(t % g8);
    int lo = 0, hi = nc;  // list l: list_off[l] <= r < list_off[l + 1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (list_off[mid] <= r) lo = mid;
        else hi = mid;
    }
    const int64_t p = xoff[lo] + (r - list_off[lo]);
    const int kb = g >> 3, e0 = (g & 7) * 8, c0 = kb * 64 + e0;
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = __float2bfloat16_rn(c0 + e < d ? X[r * dp + c0 + e] : 0.f);
    out[((((p >> 7) * (K / 64) + kb) * 128 + (p & 127)) * 64 + e0) / 8] = *reinterpret_cast<const uint4 *>(v);
}

// Squared distance (FP32) of every list row to its list's centroid, warp per row.
__global__ void row_centroid_dist_kernel(const float *__restrict__ X, int64_t n, int d, int dp,
                                         const int64_t *__restrict__ list_off, int nc, const float *__restrict__ C,
                                         float *__restrict__ out) {
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    int lo = 0, hi = nc;  // list l: list_off[l] <= r < list_off[l + 1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (list_off[mid] <= r) lo = mid;
        else hi = mid;
    }
    float s = 0.f;
    for (int t = lane; t < d; t += 32) {
        const float e = X[r * dp + t] - C[(int64_t)lo * dp + t];
        s = fmaf(e, e, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[r] = s;
}

// Inputs of the list scan's score bound (the probe stage turns them into a
// per-query bound): per list, the distances to its centroid of the 64 rows
// nearest it, ascending, each rounded up by a relative 2^-10 (covering the
// FP32 sum's rounding); +inf past the list's size.  And the largest row norm.
static int ivfl2_list_radii(IvfL2State &S, cudaStream_t st) {
    std::vector<float> dist((size_t)S.n), nrm((size_t)S.n);
    if (S.n > 0) {
        DBuf tmp;
        GN_TRY(tmp.ensure((size_t)S.n * 4));
        row_centroid_dist_kernel<<<(unsigned)ceil_div(S.n * 32, 256), 256, 0, st>>>(
            S.vecs.as<float>(), S.n, S.d, S.dp, S.list_off.as<int64_t>(), S.nc, S.cent.as<float>(), tmp.as<float>());
        GN_CUDA_TRY(cudaGetLastError());
        GN_CUDA_TRY(cudaMemcpyAsync(dist.data(), tmp.p, (size_t)S.n * 4, cudaMemcpyDeviceToHost, st));
        GN_CUDA_TRY(cudaMemcpyAsync(nrm.data(), S.vnorm.p, (size_t)S.n * 4, cudaMemcpyDeviceToHost, st));
        GN_CUDA_TRY(cudaStreamSynchronize(st));
    }
    std::vector<float> rho((size_t)S.nc * IVF_RHO, INFINITY);
    for (int32_t l = 0; l < S.nc; ++l) {
        float *b = dist.data() + S.h_off[(size_t)l], *e = dist.data() + S.h_off[(size_t)l + 1];
        const int64_t m = std::min<int64_t>(IVF_RHO, e - b);
        std::partial_sort(b, b + m, e);
        for (int64_t j = 0; j < m; ++j)
            rho[(size_t)l * IVF_RHO + j] = std::sqrt(std::max(0.f, b[j]) * (1.f + 1.f / 1024.f));
    }
    float x2 = 0.f;
    for (float v : nrm) x2 = std::max(x2, v);
    S.xmax = std::sqrt(x2 * (1.f + 1.f / 1024.f));
    GN_TRY(S.rho.ensure(rho.size() * 4));
    GN_CUDA_TRY(cudaMemcpyAsync(S.rho.p, rho.data(), rho.size() * 4, cudaMemcpyHostToDevice, st));
    GN_CUDA_TRY(cudaStreamSynchronize(st));  // rho goes out of scope
    return GN_OK;
}

int ivfl2_prepare_tc(gn_index *ix, cudaStream_t st) {
    IvfL2State &S = *ix->ivfl2;
    GN_TRY(ivfl2_list_radii(S, st));
    S.K = (int)round_up(S.d, 64);
    // BF16 list rows, tiled (see IvfL2State::x16): padded list starts
    std::vector<int64_t> xo((size_t)S.nc + 1, 0);
    for (int32_t l = 0; l < S.nc; ++l)
        xo[(size_t)l + 1] = xo[(size_t)l] + round_up(S.h_off[(size_t)l + 1] - S.h_off[(size_t)l], 128);
    S.x16_rows = std::max<int64_t>(xo[(size_t)S.nc], 128);
    if (S.x16_rows * (S.K / 64) >= ((int64_t)1 << 31))
        return fail(GN_ERR_UNSUPPORTED, "tensor-core IVF: too many rows x dimensions for the tiled layout");
    GN_TRY(S.xoff.ensure(xo.size() * 8));
    GN_CUDA_TRY(cudaMemcpyAsync(S.xoff.p, xo.data(), xo.size() * 8, cudaMemcpyHostToDevice, st));
    GN_TRY(S.x16.ensure((size_t)S.x16_rows * S.K * 2));
    GN_CUDA_TRY(cudaMemsetAsync(S.x16.p, 0, (size_t)S.x16_rows * S.K * 2, st));
    if (S.n > 0)
        x16_tiled_kernel<<<(unsigned)ceil_div(S.n * (S.K / 8), 256), 256, 0, st>>>(
            S.vecs.as<float>(), S.n, S.d, S.dp, S.list_off.as<int64_t>(), S.nc, S.xoff.as<int64_t>(), S.K,
            S.x16.as<uint4>());
    GN_CUDA_TRY(cudaStreamSynchronize(st));  // xo goes out of scope
    const int64_t crows = std::max<int64_t>(S.nc, 128);  // at least one 128-row TMA box
    GN_TRY(S.c16.ensure((size_t)crows * S.K * 2));
    GN_CUDA_TRY(cudaMemsetAsync(S.c16.p, 0, (size_t)crows * S.K * 2, st));
    to_bf16_rows(S.cent.as<float>(), S.nc, S.d, S.dp, S.c16.p, S.K, st);
    GN_TRY(S.err.ensure(4));
    GN_CUDA_TRY(cudaMemsetAsync(S.err.p, 0, 4, st));
    GN_TRY(S.sched.ensure(2 * sizeof(unsigned long long)));
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

int ivfl2_search_tc(gn_index *ix, const float *dQ, int64_t nq, int k, int64_t *d_idx, float *d_dist, int64_t *d_cnt,
                    cudaStream_t st) {
    IvfL2State &S = *ix->ivfl2;
    IvfScratch &T = S.s;
    if (k > 32 || k > S.shortlist) return fail(GN_ERR_UNSUPPORTED, "tensor-core IVF supports k <= min(32, shortlist)");
    if (S.K == 0) GN_TRY(ivfl2_prepare_tc(ix, st));
    GN_TRY(S.q16.ensure((size_t)std::max<int64_t>(nq, 256) * S.K * 2));
    to_bf16_rows(dQ, nq, S.d, S.dp, S.q16.p, S.K, st);
    int np = 1;
    GN_TRY(ivfl2_probes_tc(ix, dQ, nq, &np, st));
    // work items of rc rows (short items for small batches so that their few
    // lists still spread over all SMs); every pair owns a score segment
    const IvfL2State::TcTune &tn = S.tune[tune_bucket(nq)];
    const int rc = tn.rc ? tn.rc : (nq >= 64 ? 1024 : 256);
    // score segments in 128-row slots: slot_rel / qslot count slots, and a
    // pair's tile t has its minima at tmin4[(slot base + t) * 4 ...]
    // queries per work unit (the MMA's N side): 128, or fewer to cut a mid-size
    // batch's lists into more units
    const int qch = tn.qc ? tn.qc : TC_QCHUNK;
    GN_TRY(ivf_plan(T, nq, np, S.nc, S.list_off.as<int64_t>(), rc, qch, st, 128));
    const int64_t npairs = nq * np;
    const int64_t qb_rows = std::max<int64_t>(npairs, 256);  // >= one 256-row TMA box
    GN_TRY(S.qb.ensure((size_t)qb_rows * S.K * 2));
    GN_TRY(S.aslot.ensure((size_t)npairs * 8));
    GN_TRY(S.abound.ensure((size_t)std::max<int64_t>(npairs, 1) * 4));
    const int64_t maxlen = S.top_rows.size() > 1 ? S.top_rows[1] : 0;
    // sized for the shortest row chunk (256) so that a smaller batch never needs more
    const int64_t max_units = (ceil_div(npairs, qch) + S.nc) * (ceil_div(maxlen, 256) + 1);
    GN_TRY(S.units.ensure((size_t)max_units * sizeof(TcUnit)));
    GN_TRY(S.nunits.ensure(8));
    const unsigned qb_blocks = (unsigned)ceil_div(npairs, 8 * QB_ROWS);
    qb_units_kernel<<<qb_blocks + (unsigned)ceil_div(max_units, 256), 256, 0, st>>>(
        S.q16.as<uint4>(), S.K / 8, np, T.bucket.as<int64_t>(), T.boff.as<int64_t>(), S.nc, T.qslot.as<int64_t>(),
        T.slot_rel.as<int64_t>(), S.qb.as<uint4>(), S.aslot.as<int64_t>(), T.qbound.as<uint32_t>(),
        S.abound.as<uint32_t>(), npairs, qb_blocks,
        T.item_off.as<int64_t>(), S.list_off.as<int64_t>(), S.xoff.as<int64_t>(), rc, qch, max_units, S.units.as<TcUnit>(),
        S.nunits.as<int64_t>());
    // score slots: at most the rows of the np largest lists per query, plus one
    // partial slot per probe
    const int64_t np_eff = std::min<int64_t>(np, (int64_t)S.top_rows.size() - 1);
    const int64_t slots_total = nq * (ceil_div(S.top_rows[(size_t)np_eff], 128) + np);
    GN_TRY(S.scores.ensure((size_t)std::max<int64_t>(slots_total, 1) * 128 * 4));
    GN_TRY(S.tmin.ensure((size_t)std::max<int64_t>(slots_total, 1) * 4 * 4));
    TcIvfLaunch a;
    a.X = S.x16.p;
    a.x_rows = S.x16_rows;
    a.tiled = 1;
    a.Q = S.qb.p;
    a.q_rows = qb_rows;
    a.K = S.K;
    a.units = S.units.as<TcUnit>();
    a.n_units = S.nunits.as<int64_t>();
    a.xnorm = S.vnorm.as<float>();
    a.aslot = S.aslot.as<int64_t>();
    a.seg_mul = 128;
    a.scores = S.scores.as<float>();
    a.tmin4 = S.tmin.as<uint32_t>();
    a.abound = S.abound.as<uint32_t>();
    a.err = S.err.as<int>();
    a.next_unit = S.sched.as<unsigned long long>() + 1;
    if (S.drill) {  // armed failure drill: this launch's waits run out after ~0.1 ms
        a.drill = 1;
        a.wait_limit = 200000;
        S.drill = 0;
        S.cfg++;
    }
    a.grid = dev_info().num_sms;
    timing_begin(st, "tc_ivf_kernel");
    GN_TRY(tc_ivf_launch(a, st));
    timing_end(st);
    // selection (the tuned nt threads per query, if set)
    warps_per_query(nq, tn.nt / 32, [&](auto NWC) {
        constexpr int NW = decltype(NWC)::value;
        ivf_tc_select_kernel<NW><<<(unsigned)nq, 32 * NW, 0, st>>>(
            S.scores.as<float>(), S.tmin.as<uint4>(), T.qbound.as<uint32_t>(), T.probes.as<int32_t>(), np,
            T.qslot.as<int64_t>(), T.slot_rel.as<int64_t>(), S.list_off.as<int64_t>(), S.shortlist, dQ,
            S.vecs.as<float>(), S.d, S.dp, S.ids.as<int32_t>(), k, d_idx, d_dist, d_cnt, S.err.as<int>(),
            ix->status);
    });
    ix->status_set = ix->status != nullptr;
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

}  // namespace gn

using namespace gn;

extern "C" int gn_ivfl2_set_mode(gn_index *ix, int32_t mode, int32_t shortlist) {
    if (!ix || ix->kind != K_IVFL2 || !ix->ivfl2) return fail(GN_ERR_INVALID, "not an IVFFlatL2 index");
    if (mode != 0 && mode != 1) return fail(GN_ERR_INVALID, "mode must be 0 (FP32 scan) or 1 (tensor-core shortlist)");
    if (mode == 1 && shortlist != 16 && shortlist != 32 && shortlist != 40 && shortlist != 64)
        return fail(GN_ERR_INVALID, "shortlist must be 16, 32, 40 or 64");
    std::lock_guard<std::mutex> lk(ix->mu);
    ix->ivfl2->mode = mode;
    if (mode == 1) ix->ivfl2->shortlist = shortlist;
    ix->ivfl2->cfg++;
    return GN_OK;
}

extern "C" int gn_ivfl2_error(gn_index *ix, int32_t *err_out) {
    if (!ix || ix->kind != K_IVFL2 || !ix->ivfl2) return fail(GN_ERR_INVALID, "not an IVFFlatL2 index");
    std::lock_guard<std::mutex> lk(ix->mu);
    int herr = 0;
    if (ix->ivfl2->err.p) {
        if (ix->stream) GN_CUDA_TRY(cudaStreamSynchronize(ix->stream));
        GN_CUDA_TRY(cudaDeviceSynchronize());
        GN_CUDA_TRY(cudaMemcpy(&herr, ix->ivfl2->err.p, 4, cudaMemcpyDeviceToHost));
        if (herr) GN_CUDA_TRY(cudaMemset(ix->ivfl2->err.p, 0, 4));  // read and cleared
    }
    if (err_out) *err_out = herr;
    return GN_OK;
}

// Failure drill (tests): the next tensor-core list scan of this index issues
// no tile copies and bounds its pipeline waits to 200,000 cycles, so they run
// out: the launch ends early with the error word set and its TMEM freed.
extern "C" int gn_ivfl2_failure_drill(gn_index *ix) {
    if (!ix || ix->kind != K_IVFL2 || !ix->ivfl2) return fail(GN_ERR_INVALID, "not an IVFFlatL2 index");
    std::lock_guard<std::mutex> lk(ix->mu);
    ix->ivfl2->drill = 1;
    ix->ivfl2->cfg++;
    return GN_OK;
}

// Work of the last search (benchmark accounting; computed on demand):
// out[0] (query, probe) pairs, out[1] scored (pair, row) entries, out[2] rows
// of the distinct lists probed, out[3] tensor-core work units.
extern "C" int gn_ivfl2_last_work(gn_index *ix, int64_t *out) {
    if (!ix || ix->kind != K_IVFL2 || !ix->ivfl2) return fail(GN_ERR_INVALID, "not an IVFFlatL2 index");
    IvfL2State &S = *ix->ivfl2;
    IvfScratch &T = S.s;
    std::lock_guard<std::mutex> lk(ix->mu);
    if (!T.bcnt.p || S.nc == 0) return fail(GN_ERR_INVALID, "no search has run");
    std::vector<int32_t> cnt((size_t)S.nc);
    GN_CUDA_TRY(cudaMemcpy(cnt.data(), T.bcnt.p, (size_t)S.nc * 4, cudaMemcpyDeviceToHost));
    int64_t pairs = 0, scored = 0, rows = 0;
    for (int32_t l = 0; l < S.nc; ++l) {
        const int64_t len = S.h_off[(size_t)l + 1] - S.h_off[(size_t)l];
        pairs += cnt[(size_t)l];
        scored += (int64_t)cnt[(size_t)l] * len;
        if (cnt[(size_t)l] > 0) rows += len;
    }
    int64_t units = 0;
    if (S.mode == 1 && S.nunits.p) GN_CUDA_TRY(cudaMemcpy(&units, S.nunits.p, 8, cudaMemcpyDeviceToHost));
    out[0] = pairs;
    out[1] = scored;
    out[2] = rows;
    out[3] = units;
    return GN_OK;
}
