// flat_scan.cu — exact exhaustive k-NN scans (Hamming and float metrics).
//
// Work decomposition: the query set is cut into groups and the database into
// n_slices row slices; one CTA handles one (slice, group) unit.  Units are
// numbered slice-major so that the CTAs resident at the same time read the same
// slice and share it through L2.
//
// Hamming: hamming_append_kernel for most of an index's searches.  hamming_scan_kernel
// for those of ham_ordered, and for gn_hamming_knn_noalloc, whose partial lists have to
// fit a fixed scratch: each warp owns QW queries, lane l scores row base+l against all
// of them (query words come from shared memory as broadcasts), then offers the keys to
// the warp's register top-k lists; each (query, slice) writes its sorted k keys to a
// partial buffer, and flat_merge_kernel (flat_merge_split_kernel for small batches)
// reduces the slices.
// Float: see float_scan_kernel.  Large batches of either go to the tensor cores
// instead (tc_scan.cu).
//
// Reference semantics (pynear/include/VPTree.hpp:143-191): exact k nearest rows
// per query; here ties go to the lower row index.
#include <algorithm>

#include "distance.cuh"
#include "f32x2.cuh"
#include "flat_scan.cuh"
#include "select.cuh"
#include "tc_sm100.cuh"
#include "timing.cuh"
#include "tmap.cuh"
#include "topk.cuh"

namespace gn {

// ── Hamming scan ───────────────────────────────────────────────────────────
// db: n rows of w4 uint4 words.  q: nq rows, same layout.
template <int QW, int R>
__global__ void __launch_bounds__(128) hamming_scan_kernel(const uint4 *__restrict__ db, int64_t n, int w4,
                                                           const uint4 *__restrict__ q, int64_t nq, int k,
                                                           int n_slices, int64_t slice_rows, int n_groups,
                                                           uint64_t *__restrict__ part) {
    extern __shared__ uint4 sq[];  // [WARPS*QW][w4]
    const int warps = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.x;
    const int slice = unit / n_groups, group = unit % n_groups;
    const int64_t q0 = (int64_t)group * warps * QW;

    for (int i = threadIdx.x; i < warps * QW * w4; i += blockDim.x) {
        int64_t qi = q0 + i / w4;
        sq[i] = (qi < nq) ? q[qi * w4 + (i % w4)] : make_uint4(0, 0, 0, 0);
    }
    __syncthreads();

    const int64_t r0 = (int64_t)slice * slice_rows;
    const int64_t r1 = min(n, r0 + slice_rows);
    const uint4 *myq = sq + warp * QW * w4;

    WarpTopK<R> lists[QW];
    uint64_t thr[QW];
#pragma unroll
    for (int j = 0; j < QW; ++j) { lists[j].init(); thr[j] = KEY_EMPTY; }

    for (int64_t base = r0; base < r1; base += 32) {
        const int64_t row = base + lane;
        const bool valid = row < r1;
        uint32_t dist[QW];
#pragma unroll
        for (int j = 0; j < QW; ++j) dist[j] = 0;
        const uint4 *rp = db + (valid ? row : r0) * w4;
#pragma unroll 4
        for (int c = 0; c < w4; ++c) {
            uint4 x = ldg_nc_u4(rp + c);
#pragma unroll
            for (int j = 0; j < QW; ++j) dist[j] += popc4(x, myq[j * w4 + c]);
        }
#pragma unroll
        for (int j = 0; j < QW; ++j) {
            uint64_t key = valid ? make_key(dist[j], (uint32_t)row) : KEY_EMPTY;
            lists[j].offer(key, thr[j], k);
        }
    }
#pragma unroll
    for (int j = 0; j < QW; ++j) {
        int64_t qi = q0 + warp * QW + j;
        if (qi < nq) lists[j].store(part + ((size_t)qi * n_slices + slice) * k, k);
    }
}

// ── float scan (L2 / L1 / Linf in the reference's arithmetic order) ───────
// db: n rows of dp floats (dp % 4 == 0, zero padded past d).
//
// A unit is (row slice, query group).  Four warps: WQ across the group's
// queries (QW each), WR = 4 / WQ across a stage's rows; a lane scores RPT rows
// against the warp's QW queries at a time, each (row, query) pair whole in one
// thread (the reference's eight-accumulator order needs it), so a row's 16-byte
// shared load serves QW queries and a query's broadcast RPT rows.  Arithmetic is
// packed FP32 (f32x2.cuh) on row + (-query): the squares and magnitudes are those
// of query - row bit for bit.
//
// Rows reach shared memory by TMA (cp.async.bulk.tensor) in boxes of 32 floats
// (128 bytes) x the stage's rows with the 128-byte swizzle, so the 16-byte chunk
// c of row r sits at chunk c ^ (r & 7) of the row's 128 bytes and the eight lanes
// of each quarter-warp phase of a 16-byte shared load (eight consecutive rows,
// same logical chunk) hit eight different bank groups.  Thread 0 keeps
// FS_STAGES - 1 stages in flight ahead of the one consumed (one mbarrier per
// stage in each direction, bounded waits; the warps may be a stage apart).
//
// Selection: a pair that can still be among its list's k nearest is appended to
// the list's buffer of `cap` keys without order (one ballot); a full buffer is
// cut down to its k best by counting (select.cuh), which also lowers the list's
// threshold.  An ordered register list took ~300 cycles per insertion and, for
// k = 100 over 11 slices, 95 % of the scan.  At the end of its slice a list adds
// its k best to the query's candidates, from which flat_finish_kernel takes the
// answer.
//
// Measured, scan alone (before: one row per lane and four queries per warp in
// scalar arithmetic, ordered lists): 100k x 32, 1,000 queries, k 5: 519 -> 416 us
// (FP32 pipe 41 % busy; floor 159 us); L1 over 30,011 x 97, 513 queries, k 100:
// 1611 -> 284 us (floor 74 us); 1M x 128, 8 queries: 180 -> 166 us (512 MB, 76 us
// of HBM time); 20k x 64, 1 query: 14.9 -> 7.7 us.
constexpr int FS_BOX = 32;      // floats per box row (128 bytes)
constexpr int FS_STAGES = 3;
constexpr int FS_STAGE = 16384; // bytes of a stage at most
constexpr int FS_THREADS = 128, FS_WARPS = 4;

// Launch shape of a batch.
struct FsGeom {
    int qw, rpt, wq, wr;  // queries per warp, rows per lane, warps across queries and rows
    int nbx, bw;          // boxes per row, floats per box row: 32 (swizzled) or the row width (narrow rows)
    int rows, cb, nchunk; // rows and boxes per stage, column chunks per row
    int cap, most;        // keys of a list's buffer, and how many it may hold before it is cut
    size_t smem;
};

static FsGeom fs_geom(int64_t n, int64_t nq, int k, int dp4) {
    FsGeom g;
    g.cap = list_cap(k);  // k <= 64: in shared memory, else in global
    g.most = list_most(k);
    // small batches: one or two queries per warp, every warp on its own rows; from
    // five queries on a row's load serves four of them
    g.qw = nq <= 1 ? 1 : nq <= 2 ? 2 : 4;
    g.wq = nq <= 4 ? 1 : nq <= 8 ? 2 : 4;
    // the queries must fit beside the ring and the buffers
    auto qbytes = [&]() { return (size_t)g.wq * g.qw * dp4 * 16; };
    while (qbytes() > 100 * 1024 && g.wq > 1) g.wq >>= 1;
    while (qbytes() > 130 * 1024 && g.qw > 1) g.qw >>= 1;
    // (several warps across the queries: four queries each; up to 32 rows fill one per lane)
    g.rpt = g.wq > 1 && n > 32 ? 2 : 1;
    g.wr = FS_WARPS / g.wq;
    // rows the four warps take at a time, no more than there are: a stage of fewer rows
    // has room for more boxes of each
    const int unit = (int)std::min<int64_t>(32 * g.rpt * g.wr, round_up(std::max<int64_t>(n, 1), 32 * g.rpt));
    g.nbx = (dp4 * 4 + FS_BOX - 1) / FS_BOX;
    g.bw = dp4 * 4 < FS_BOX ? dp4 * 4 : FS_BOX;
    g.cb = std::min(g.nbx, std::max(1, FS_STAGE / (unit * 128)));
    g.nchunk = (g.nbx + g.cb - 1) / g.cb;
    g.rows = unit;
    if (g.nchunk == 1)  // short rows: more of them per stage (a TMA box has at most 256 rows)
        while (g.rows * 2 <= 256 && (size_t)g.rows * 2 * g.cb * g.bw * 4 <= FS_STAGE) g.rows *= 2;
    g.smem = qbytes() + 1024 + (size_t)FS_STAGES * g.cb * g.rows * g.bw * 4 + FS_STAGES * 16 +
             (g.cap == LIST_CAP_S ? (size_t)FS_WARPS * g.qw * LIST_CAP_S * 8 : 0);
    return g;
}

struct FsArgs {
    int64_t n, nq, slice_rows, list_keys;
    int d, dp4, k, n_slices, n_groups;
    int wq, wr, nbx, bw, rows, cb, nchunk, cap, most;
    const float *q;
    uint64_t *gbuf;  // buffers of k > 64: per CTA, warp and query, cap keys
    uint64_t *cand;  // per query list_keys candidate keys ...
    int *qcount;     // ... and how many there are
    int *err;
    const int *only_if;
};

// One (row, query) pair's accumulators: the packed form of distance.cuh's FAcc.
template <int METRIC>
struct FPair {
    f32x2 p[4];  // L2: lanes (0, 1) (2, 3) (4, 5) (6, 7); else unused
    float a[8];  // L1, Linf
    __device__ __forceinline__ void zero() {
        if (METRIC == M_L2) {
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = 0ull;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = 0.f;
        }
    }
    // eight coordinates: x the row's, m the query's negated
    __device__ __forceinline__ void block8(const f32x2 (&x)[4], const f32x2 (&m)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const f32x2 t = add2(x[i], m[i]);
            if (METRIC == M_L2) {
                p[i] = fma2(t, t, p[i]);
            } else {
                float lo, hi;
                unpack2(t, lo, hi);
                if (METRIC == M_L1) {
                    a[2 * i] = __fadd_rn(a[2 * i], fabsf(lo));
                    a[2 * i + 1] = __fadd_rn(a[2 * i + 1], fabsf(hi));
                } else {
                    a[2 * i] = fmaxf(a[2 * i], fabsf(lo));
                    a[2 * i + 1] = fmaxf(a[2 * i + 1], fabsf(hi));
                }
            }
        }
    }
    // After the blocks of eight, in FAcc::finish's order: fold, then for d % 8 = rem
    // coordinates left (q0, q1 and x0, x1, the query's negated, zero past d) tail,
    // then value: what orders rows as the distance does, for L2 the squared sum
    // under the root, else the distance.
    __device__ __forceinline__ void fold() {
        if (METRIC == M_L2) {
            p[0] = add2(p[2], p[0]);
            p[1] = add2(p[3], p[1]);
        } else {
#pragma unroll
            for (int i = 1; i < 8; ++i) a[0] = METRIC == M_L1 ? __fadd_rn(a[0], a[i]) : fmaxf(a[0], a[i]);
        }
    }
    __device__ __forceinline__ void tail(int rem, const float4 &q0, const float4 &q1, const float4 &x0,
                                         const float4 &x1) {
        const float t[8] = {__fadd_rn(x0.x, q0.x), __fadd_rn(x0.y, q0.y), __fadd_rn(x0.z, q0.z),
                            __fadd_rn(x0.w, q0.w), __fadd_rn(x1.x, q1.x), __fadd_rn(x1.y, q1.y),
                            __fadd_rn(x1.z, q1.z), __fadd_rn(x1.w, q1.w)};
        if (METRIC == M_L2) {
            const f32x2 t01 = pack2(t[0], t[1]), t23 = pack2(t[2], t[3]);
            p[0] = fma2(t01, t01, p[0]);
            p[1] = fma2(t23, t23, p[1]);
            if (rem > 4) {
                const f32x2 t45 = pack2(t[4], t[5]), t67 = pack2(t[6], t[7]);
                p[0] = fma2(t45, t45, p[0]);
                p[1] = fma2(t67, t67, p[1]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 7; ++i)
                if (i < rem) a[0] = METRIC == M_L1 ? __fadd_rn(a[0], fabsf(t[i])) : fmaxf(a[0], fabsf(t[i]));
        }
    }
    __device__ __forceinline__ float value() const {
        if (METRIC != M_L2) return a[0];
        float s0, s1, s2, s3;
        unpack2(p[0], s0, s1);
        unpack2(p[1], s2, s3);
        return __fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2, s3));
    }
};

// The largest finish() value (as bits) of a distance below thr: L2, a squared sum
// above thr * thr (rounded up) has a root of at least thr, so the root itself is
// taken only for rows that may enter.
template <int METRIC>
__device__ __forceinline__ uint32_t fs_limit(uint32_t thr) {
    if (METRIC != M_L2 || thr >= 0x7f800000u) return thr;  // no bound yet, or one that is not finite
    const float t = __uint_as_float(thr);
    return __float_as_uint(__fmul_ru(t, t));
}

// list_add for finish() bits v, as a call (see list_cut): L2 takes the root here.
template <int METRIC>
__device__ __noinline__ uint2 fs_add(uint64_t *buf, uint2 state, uint32_t v, bool in, uint32_t row, int k, int most) {
    if (METRIC == M_L2) v = __float_as_uint(__fsqrt_rn(__uint_as_float(v)));
    return list_add<true>(buf, state, v, in, row, k, most);
}

// ONE: a stage holds whole rows (the accumulators then never outlive a group).
template <int METRIC, int QW, int RPT, bool ONE>
__global__ void __launch_bounds__(FS_THREADS, 3)
    float_scan_kernel(const __grid_constant__ CUtensorMap tm, const FsArgs a) {
    if (a.only_if && *a.only_if == 0) return;
    extern __shared__ float4 sqf[];  // [WQ * QW][dp4] negated queries, buffers (k <= 64), the stage ring, barriers
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slice = blockIdx.x / a.n_groups, group = blockIdx.x % a.n_groups;
    const int wqi = warp % a.wq, wri = warp / a.wq;
    const int64_t q0 = (int64_t)group * a.wq * QW;
    const int dp4 = a.dp4, k = a.k;
    uint64_t *sbuf = reinterpret_cast<uint64_t *>(sqf + a.wq * QW * dp4);
    const int cap = a.cap;
    // (an offset from the shared array, not a rounded pointer: the loads stay shared-memory loads)
    const uint32_t ring_at = (uint32_t)(a.wq * QW * dp4) * 16 + (cap == LIST_CAP_S ? FS_WARPS * QW * LIST_CAP_S * 8 : 0);
    const uint32_t smem0 = smem_u32(sqf);
    uint8_t *ring = reinterpret_cast<uint8_t *>(sqf) + (((smem0 + ring_at + 1023) & ~1023u) - smem0);
    const uint32_t pitch = (uint32_t)a.bw * 4, box_bytes = (uint32_t)a.rows * pitch;
    const uint32_t stage_bytes = (uint32_t)a.cb * box_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + FS_STAGES * stage_bytes);
    volatile int *verr = a.err;

    const float4 *q4 = reinterpret_cast<const float4 *>(a.q);
    for (int i = threadIdx.x; i < a.wq * QW * dp4; i += FS_THREADS) {
        const int64_t qi = q0 + i / dp4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (qi < a.nq) v = q4[qi * dp4 + (i % dp4)];
        sqf[i] = make_float4(-v.x, -v.y, -v.z, -v.w);
    }
    uint64_t *empty = full + FS_STAGES;
    if (threadIdx.x == 0) {
        for (int s = 0; s < FS_STAGES; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, FS_WARPS);
        }
        mbar_fence_init();
    }

    const int64_t r0 = (int64_t)slice * a.slice_rows;
    const int64_t r1 = min(a.n, r0 + a.slice_rows);
    const float4 *myq = sqf + wqi * QW * dp4;
    const int nb = a.d >> 3, rem = a.d & 7;
    const int nstage = (int)((r1 - r0 + a.rows - 1) / a.rows) * a.nchunk;

    // stages in order (row group, then its column chunks) into ring slots in turn; the
    // issuing thread's place in that order
    int iss = 0, iss_slot = 0, iss_y = (int)r0, iss_b0 = 0;
    uint32_t iss_ph = 0;  // parity of the release that frees the slot: its use before
    auto issue = [&]() {
        const int nbox = min(a.cb, a.nbx - iss_b0);
        uint8_t *dst = ring + (uint32_t)iss_slot * stage_bytes;
        mbar_expect_tx(full + iss_slot, (uint32_t)nbox * box_bytes);
        for (int bi = 0; bi < nbox; ++bi)
            tma_load_2d(dst + bi * box_bytes, &tm, (iss_b0 + bi) * a.bw, iss_y, full + iss_slot);
        ++iss;
        iss_b0 += a.cb;
        if (ONE || iss_b0 >= a.nbx) {
            iss_b0 = 0;
            iss_y += a.rows;
        }
        if (++iss_slot == FS_STAGES) {
            iss_slot = 0;
            iss_ph ^= 1;
        }
    };

    // a list: its buffer, the keys in it, and the distance bits that a new key must
    // stay below (rows come in ascending order, so an equal distance loses the tie)
    uint64_t *buf0 = cap == LIST_CAP_S ? sbuf + warp * QW * LIST_CAP_S
                                     : a.gbuf + ((size_t)blockIdx.x * FS_WARPS + warp) * QW * cap;
    int cnt[QW];
    uint32_t thr[QW], lim[QW];  // lim: fs_limit(thr)
#pragma unroll
    for (int j = 0; j < QW; ++j) {
        cnt[j] = 0;
        thr[j] = lim[j] = q0 + wqi * QW + j < a.nq ? 0xffffffffu : 0u;
    }
    __syncthreads();  // queries and barriers ready
    if (threadIdx.x == 0)
        while (iss < min(FS_STAGES - 1, nstage)) issue();
    const uint32_t sw = a.bw < FS_BOX ? 0u : (uint32_t)(lane & 7);  // a lane's rows are lane modulo 32
    uint32_t off[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) off[c] = ((uint32_t)c ^ sw) << 4;
    const int wrows = 32 * RPT;  // rows a warp takes at a time
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    FPair<METRIC> acc[RPT][QW];
    bool ok = true;
    int slot = 0, kc = 0;
    uint32_t ph = 0;
    int si = 0;
    int64_t y0 = r0;
    for (; si < nstage; ++si) {
        // keep FS_STAGES - 1 stages in flight: the next goes to the slot of stage si - 1,
        // once every warp has left that (the warps may be a stage apart)
        if (threadIdx.x == 0 && iss < nstage) {
            if (iss >= FS_STAGES && !mbar_wait(empty + iss_slot, iss_ph ^ 1, verr)) ok = false;
            else issue();
        }
        if (!__all_sync(0xffffffffu, ok && mbar_wait(full + slot, ph, verr))) {
            ok = false;
            break;
        }
        const uint8_t *st = ring + (size_t)slot * stage_bytes;
        const int b0 = kc * a.cb, nbox = min(a.cb, a.nbx - b0);
        const bool last = ONE || kc == a.nchunk - 1;
        for (int g = wri * wrows; g < a.rows; g += a.wr * wrows) {
            if (y0 + g >= r1) break;
            const uint8_t *rp[RPT];
#pragma unroll
            for (int r = 0; r < RPT; ++r) rp[r] = st + (uint32_t)(g + r * 32 + lane) * pitch;
            if (ONE || kc == 0) {
#pragma unroll
                for (int r = 0; r < RPT; ++r)
#pragma unroll
                    for (int j = 0; j < QW; ++j) acc[r][j].zero();
            }
            // coordinates 8 e .. of the box at boff; o0, o1: its two chunks' offsets in a row
            auto eight = [&](uint32_t boff, const float4 *qb, uint32_t o0, uint32_t o1, int e) {
                f32x2 x[RPT][4];
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    const ulonglong2 lo = *reinterpret_cast<const ulonglong2 *>(rp[r] + boff + o0);
                    const ulonglong2 hi = *reinterpret_cast<const ulonglong2 *>(rp[r] + boff + o1);
                    x[r][0] = lo.x;
                    x[r][1] = lo.y;
                    x[r][2] = hi.x;
                    x[r][3] = hi.y;
                }
#pragma unroll
                for (int j = 0; j < QW; ++j) {
                    const ulonglong2 lo = *reinterpret_cast<const ulonglong2 *>(qb + j * dp4 + 2 * e);
                    const ulonglong2 hi = *reinterpret_cast<const ulonglong2 *>(qb + j * dp4 + 2 * e + 1);
                    const f32x2 m[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
                    for (int r = 0; r < RPT; ++r) acc[r][j].block8(x[r], m);
                }
            };
            // whole boxes, then the blocks of eight of a partial one
            const int blocks = min(nb - b0 * 4, nbox * 4), whole = blocks >> 2;
            for (int bi = 0; bi < whole; ++bi) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    eight((uint32_t)bi * box_bytes, myq + (b0 + bi) * 8, off[2 * e], off[2 * e + 1], e);
            }
#pragma unroll 1
            for (int e = 0; e < blocks - whole * 4; ++e)
                eight((uint32_t)whole * box_bytes, myq + (b0 + whole) * 8, ((uint32_t)(2 * e) ^ sw) << 4,
                      ((uint32_t)(2 * e + 1) ^ sw) << 4, e);
            if (!last) continue;
            const int left = (int)min((int64_t)a.rows, r1 - y0) - g;  // rows from this group on
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
#pragma unroll
                for (int j = 0; j < QW; ++j) acc[r][j].fold();
            }
            if (rem > 0) {  // the remainder's coordinates sit in the last box
                const int tail4 = 2 * nb;
                const uint32_t tb = (uint32_t)((tail4 >> 3) - b0) * box_bytes;
                const uint32_t o0 = ((uint32_t)(tail4 & 7) ^ sw) << 4, o1 = ((uint32_t)((tail4 & 7) + 1) ^ sw) << 4;
                const float4 *tq = myq + tail4;
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    const float4 x0 = *reinterpret_cast<const float4 *>(rp[r] + tb + o0);
                    const float4 x1 = rem > 4 ? *reinterpret_cast<const float4 *>(rp[r] + tb + o1) : zero4;
#pragma unroll
                    for (int j = 0; j < QW; ++j)
                        acc[r][j].tail(rem, tq[j * dp4], rem > 4 ? tq[j * dp4 + 1] : zero4, x0, x1);
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                uint32_t bits[QW];
                bool any = false;
#pragma unroll
                for (int j = 0; j < QW; ++j) {
                    bits[j] = __float_as_uint(acc[r][j].value());
                    any = any || bits[j] <= lim[j];
                }
                if (!__any_sync(0xffffffffu, any)) continue;
                const uint32_t row = (uint32_t)(y0 + g) + r * 32 + lane;
#pragma unroll
                for (int j = 0; j < QW; ++j) {
                    const bool in = bits[j] <= lim[j] && r * 32 + lane < left;
                    if (!__any_sync(0xffffffffu, in)) continue;
                    const uint2 ns = fs_add<METRIC>(buf0 + j * cap, make_uint2(cnt[j], thr[j]), bits[j], in, row, k,
                                                    a.most);
                    cnt[j] = (int)ns.x;
                    if (ns.y != thr[j]) {
                        thr[j] = ns.y;
                        lim[j] = fs_limit<METRIC>(ns.y);
                    }
                }
            }
        }
        if (ONE || ++kc == a.nchunk) {
            kc = 0;
            y0 += a.rows;
        }
        mbar_release_warp(empty + slot);
        if (++slot == FS_STAGES) {
            slot = 0;
            ph ^= 1;
        }
    }
    if (!ok) {
        // a wait ran out in stage si (the other warps find the error word set, or run
        // out themselves): let the copies issued from stage si on land (each wait bounded)
        // before the issuing thread leaves
        if (threadIdx.x == 0)
            for (int x = si; x < iss; ++x) {
                const long long t0 = clock64();
                while (!mbar_try_wait(full + x % FS_STAGES, (uint32_t)((x / FS_STAGES) & 1)) &&
                       clock64() - t0 < 400000) {
                }
            }
        return;
    }
#pragma unroll
    for (int j = 0; j < QW; ++j) {
        const int64_t qi = q0 + wqi * QW + j;
        if (qi >= a.nq) continue;
        uint64_t *b = buf0 + j * cap;
        int c = cnt[j];
        if (c > k) {
            list_cut_k(b, c, k);
            c = k;
        }
        __syncwarp();
        int at = 0;
        if (lane == 0) at = atomicAdd(a.qcount + qi, c);
        at = __shfl_sync(0xffffffffu, at, 0);
        uint64_t *dst = a.cand + qi * a.list_keys + at;
        for (int i = lane; i < c; i += 32) dst[i] = b[i];
    }
}

// ── exact Hamming, appended candidates ────────────────────────────────────
__device__ __noinline__ uint2 ham_add(uint64_t *buf, uint2 state, uint32_t dist, bool in, uint32_t row, int k,
                                      int most) {
    return list_add<true>(buf, state, dist, in, row, k, most);
}

// One CTA per (slice of rows, group of wq QW queries): lane = RPT rows, QW queries a
// warp, broadcast from shared memory, the CTA's four warps wq across the queries and
// 4 / wq across the rows (a list that sees four times the rows takes few more of them:
// with every warp on its own rows, taking candidates was two thirds of the
// instructions).  A row below its
// query's threshold is appended to the warp's buffer, which is cut to its k best by
// counting when it fills (list_add); at the end of the slice the k best go to the query's
// candidates, from which flat_finish_kernel takes the answer.  A cut's k-th distance is
// also a bound for the query's other lists, up to and including it: the lowest stands,
// inverted (so that zero is none), in bound[q], read with each step's rows.
// Eight words of a row are run together by carry-save addition, so that the counts
// (POPC) are half of what they were.  Whole searches of 1M x 512 bits, before (a register
// list in order per query, eight queries a warp, four warps of queries whatever the
// batch) and now: 1 query 326 -> 65 us, 16: 335 -> 139, 100: 670 -> 516, 100 with k 90:
// 4161 -> 659; 20k x 512 bits, 3,000 queries: 416 -> 334.
constexpr int HAM_CTAS = 5;  // per SM (102 registers a thread)
template <int QW, int RPT>
__global__ void __launch_bounds__(128, HAM_CTAS)
    hamming_append_kernel(const uint4 *__restrict__ db, int64_t n, int w4, const uint4 *__restrict__ q, int64_t nq,
                          int k, int cap, int most, int wq, int64_t slice_rows, int n_groups,
                          uint64_t *__restrict__ cand,
                          int64_t list_keys, int *__restrict__ qcount, uint32_t *bound) {
    extern __shared__ uint4 sqs[];  // [wq QW][w4], then the buffers [4][QW][cap]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slice = blockIdx.x / n_groups, group = blockIdx.x % n_groups;
    const int wr = 4 / wq, wri = warp / wq;
    const int64_t g0 = (int64_t)group * wq * QW, q0 = g0 + (warp % wq) * QW;
    for (int i = threadIdx.x; i < wq * QW * w4; i += 128)
        sqs[i] = g0 + i / w4 < nq ? q[g0 * w4 + i] : make_uint4(0u, 0u, 0u, 0u);
    const uint4 *const sq = sqs + (warp % wq) * QW * w4;
    uint64_t *const buf0 = reinterpret_cast<uint64_t *>(sqs + wq * QW * w4) + (size_t)warp * QW * cap;
    int cnt[QW];
    uint32_t thr[QW];
#pragma unroll
    for (int j = 0; j < QW; ++j) {
        cnt[j] = 0;
        thr[j] = q0 + j < nq ? 0xffffffffu : 0u;
    }
    __syncthreads();
    const int64_t r0 = (int64_t)slice * slice_rows, r1 = min(n, r0 + slice_rows);
    if (q0 >= nq) return;  // (no barrier follows)
    for (int64_t base = r0 + wri * 32 * RPT; base < r1; base += wr * 32 * RPT) {
        const uint4 *rp[RPT];
        uint32_t dist[RPT][QW];
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            rp[r] = db + min(base + r * 32 + lane, r1 - 1) * w4;
#pragma unroll
            for (int j = 0; j < QW; ++j) dist[r][j] = 0;
        }
        uint32_t all = 0xffffffffu;  // lane j: query j's bound
        if (lane < QW && q0 + lane < nq) all = ~*reinterpret_cast<volatile uint32_t *>(bound + q0 + lane);
        int c = 0;
#pragma unroll 2
        for (; c + 1 < w4; c += 2) {
            uint4 x0[RPT], x1[RPT];
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                x0[r] = ldg_nc_u4(rp[r] + c);
                x1[r] = ldg_nc_u4(rp[r] + c + 1);
            }
#pragma unroll
            for (int j = 0; j < QW; ++j) {
                const uint4 a = sq[j * w4 + c], b = sq[j * w4 + c + 1];
#pragma unroll
                for (int r = 0; r < RPT; ++r) dist[r][j] += popc8(x0[r], a, x1[r], b);
            }
        }
        if (c < w4) {
            uint4 x[RPT];
#pragma unroll
            for (int r = 0; r < RPT; ++r) x[r] = ldg_nc_u4(rp[r] + c);
#pragma unroll
            for (int j = 0; j < QW; ++j) {
                const uint4 a = sq[j * w4 + c];
#pragma unroll
                for (int r = 0; r < RPT; ++r) dist[r][j] += popc4(x[r], a);
            }
        }
#pragma unroll
        for (int j = 0; j < QW; ++j) thr[j] = min(thr[j], __shfl_sync(0xffffffffu, all, j));
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int64_t row = base + r * 32 + lane;
#pragma unroll
            for (int j = 0; j < QW; ++j) {
                const bool in = row < r1 && dist[r][j] < thr[j];
                if (!__any_sync(0xffffffffu, in)) continue;
                const uint2 st = ham_add(buf0 + j * cap, make_uint2(cnt[j], thr[j]), dist[r][j], in, (uint32_t)row, k,
                                         most);
                cnt[j] = (int)st.x;
                if (st.y != thr[j] && lane == 0) atomicMax(bound + q0 + j, ~(st.y + 1u));
                thr[j] = st.y;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < QW; ++j) {
        const int64_t qi = q0 + j;
        int m = cnt[j];
        if (qi >= nq || m == 0) continue;
        uint64_t *b = buf0 + j * cap;
        if (m > k) {
            list_cut_k(b, m, k);
            m = k;
        }
        __syncwarp();
        int at = 0;
        if (lane == 0) at = atomicAdd(qcount + qi, m);
        at = __shfl_sync(0xffffffffu, at, 0);
        uint64_t *dst = cand + qi * list_keys + at;
        for (int i = lane; i < m; i += 32) dst[i] = b[i];
    }
}

// The answer from a query's candidates: each of the block's W warps takes the k
// best of its share, the first warp the k best of theirs, sorted.  One warp per
// query where the batch alone fills the GPU, 8 or 24 for smaller batches, whose
// queries have hundreds of lists each.
template <int W, int R, typename Dist = float>
__global__ void __launch_bounds__(W * 32)
    flat_finish_kernel(const uint64_t *__restrict__ cand, const int *__restrict__ qcount, int64_t list_keys, int k,
                       int64_t *__restrict__ out_idx, Dist *__restrict__ out_dist, int64_t *__restrict__ out_cnt,
                       const int *__restrict__ only_if, const int *err, int *status) {
    __shared__ uint64_t s_sel[(W + 1) * R * 32];
    __shared__ int s_n[W];
    if (status && blockIdx.x == 0 && threadIdx.x == 0) *status = *err;
    if (only_if && *only_if == 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t q = blockIdx.x;
    const uint64_t *p = cand + q * list_keys;
    const int total = qcount[q];
    const int share = (total + W - 1) / W;
    const int b = min(total, warp * share), e = min(total, b + share);
    const int mine = warp_best(p + b, e - b, k, s_sel + warp * R * 32);
    uint64_t *res = s_sel;
    int m = mine;
    if (W > 1) {
        if (lane == 0) s_n[warp] = mine;
        __syncthreads();
        if (warp != 0) return;
        // the warps' keys, moved together (each group moves down, in order)
        m = mine;
        for (int w = 1; w < W; ++w) {
            const int nw = s_n[w];
            for (int i = 0; i < nw; i += 32) {
                const uint64_t key = i + lane < nw ? s_sel[w * R * 32 + i + lane] : 0ull;
                __syncwarp();
                if (i + lane < nw) s_sel[m + i + lane] = key;
                __syncwarp();
            }
            m += nw;
        }
        res = s_sel + W * R * 32;
        m = warp_best(s_sel, m, k, res);
    }
    if (out_cnt && lane == 0) out_cnt[q] = m;
    uint64_t v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = r * 32 + lane < m ? res[r * 32 + lane] : KEY_EMPTY;
    warp_sort<R>(v);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int pos = r * 32 + lane;
        if (pos >= k) continue;
        const bool empty = v[r] == KEY_EMPTY;
        out_idx[q * k + pos] = empty ? -1 : (int64_t)key_idx(v[r]);
        if constexpr (sizeof(Dist) == 8) out_dist[q * k + pos] = empty ? 0 : (Dist)key_dist(v[r]);
        else out_dist[q * k + pos] = empty ? 0.f : __uint_as_float(key_dist(v[r]));
    }
}

// ── Hamming scan: merge of per-slice partial lists → final output ─────────
// Offer a query's sorted per-slice lists s_begin, s_begin + s_step, ... (k <=
// 32: one 32-key chunk per slice) to a warp's list: the chunks of MERGE_AHEAD
// slices are loaded together, so that a small batch's hundreds of slices cost
// hundreds / MERGE_AHEAD load latencies instead of one each.
constexpr int MERGE_AHEAD = 16;
template <int R>
__device__ __forceinline__ void merge_slices_ahead(const uint64_t *__restrict__ p, int s_begin, int n_slices,
                                                   int s_step, int k, int lane, WarpTopK<R> &L, uint64_t &thr) {
    for (int s0 = s_begin; s0 < n_slices; s0 += MERGE_AHEAD * s_step) {
        uint64_t kk[MERGE_AHEAD];
#pragma unroll
        for (int u = 0; u < MERGE_AHEAD; ++u) {
            const int s = s0 + u * s_step;
            kk[u] = (s < n_slices && lane < k) ? p[(size_t)s * k + lane] : KEY_EMPTY;
        }
#pragma unroll
        for (int u = 0; u < MERGE_AHEAD; ++u)
            if (!__all_sync(0xffffffffu, kk[u] >= thr)) L.offer(kk[u], thr, k);
    }
}

// Write a query's k nearest: idx (-1 for empty) and distance.
template <int R>
__device__ __forceinline__ void merge_store(const WarpTopK<R> &L, int64_t qi, int k, int lane,
                                            int64_t *__restrict__ out_idx, int64_t *__restrict__ out_dist) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int pos = r * 32 + lane;
        if (pos < k) {
            uint64_t key = L.v[r];
            bool e = key == KEY_EMPTY;
            out_idx[qi * k + pos] = e ? -1 : (int64_t)key_idx(key);
            out_dist[qi * k + pos] = e ? 0 : (int64_t)key_dist(key);
        }
    }
}

// One warp per query.
template <int R>
__global__ void flat_merge_kernel(const uint64_t *__restrict__ part, int n_slices, int k, int64_t nq,
                                  int64_t *__restrict__ out_idx, int64_t *__restrict__ out_dist) {
    const int lane = threadIdx.x & 31;
    const int64_t qi = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (qi >= nq) return;
    WarpTopK<R> L;
    L.init();
    uint64_t thr = KEY_EMPTY;
    const uint64_t *p = part + (size_t)qi * n_slices * k;
    if (k <= 32) merge_slices_ahead(p, 0, n_slices, 1, k, lane, L, thr);
    else for (int s = 0; s < n_slices; ++s) {
        for (int j0 = 0; j0 < k; j0 += 32) {
            int j = j0 + lane;
            uint64_t key = (j < k) ? p[(size_t)s * k + j] : KEY_EMPTY;
            // partial lists are sorted: once the smallest unseen key of this
            // chunk is above the threshold the rest of the list is too
            if (__all_sync(0xffffffffu, key >= thr)) break;
            L.offer(key, thr, k);
        }
    }
    merge_store(L, qi, k, lane, out_idx, out_dist);
}

// Small batches (k <= 32): one block of MERGE_WARPS warps per query, so that
// a batch too small to fill the GPU with one warp per query still merges its
// hundreds of slices quickly: warp w takes slices w, w + MERGE_WARPS, ...,
// then warp 0 offers the other warps' first k keys (disjoint rows) to its own
// list.  The k nearest are the same keys in the same order as flat_merge_kernel's.
constexpr int MERGE_WARPS = 8;
__global__ void __launch_bounds__(MERGE_WARPS * 32)
    flat_merge_split_kernel(const uint64_t *__restrict__ part, int n_slices, int k, int64_t *__restrict__ out_idx,
                            int64_t *__restrict__ out_dist) {
    __shared__ uint64_t wl[MERGE_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t qi = blockIdx.x;
    WarpTopK<1> L;
    L.init();
    uint64_t thr = KEY_EMPTY;
    merge_slices_ahead(part + (size_t)qi * n_slices * k, warp, n_slices, MERGE_WARPS, k, lane, L, thr);
    wl[warp][lane] = lane < k ? L.v[0] : KEY_EMPTY;
    __syncthreads();
    if (warp != 0) return;
#pragma unroll 1
    for (int w = 1; w < MERGE_WARPS; ++w) {
        const uint64_t key = wl[w][lane];
        if (!__all_sync(0xffffffffu, key >= thr)) L.offer(key, thr, k);
    }
    merge_store(L, qi, k, lane, out_idx, out_dist);
}

// ── large-k path: materialised keys + radix select + bitonic sort ────────
template <int METRIC>
__global__ void flat_keys_kernel(const void *__restrict__ db, int64_t n, int d, int stride4,
                                 const void *__restrict__ q, int64_t q_begin, int64_t qc,
                                 uint64_t *__restrict__ keys) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t qq = t / n, row = t % n;
    if (qq >= qc) return;
    const int64_t qi = q_begin + qq;
    uint32_t bits;
    if (METRIC == M_HAMMING) {
        bits = hdist(reinterpret_cast<const uint4 *>(q) + qi * stride4, reinterpret_cast<const uint4 *>(db) + row * stride4,
                     stride4);
    } else {
        bits = __float_as_uint(fdist<METRIC>(reinterpret_cast<const float *>(q) + qi * stride4 * 4,
                                             reinterpret_cast<const float *>(db) + row * stride4 * 4, d));
    }
    keys[qq * n + row] = make_key(bits, (uint32_t)row);
}

// One CTA per query: exact k-th smallest key by MSD radix select (8-bit
// digits), gather the k keys at or below it, bitonic-sort them in place.
__global__ void __launch_bounds__(1024) radix_select_sort_kernel(const uint64_t *__restrict__ keys, int64_t n,
                                                                 int64_t k, int64_t pow2,
                                                                 uint64_t *__restrict__ sorted) {
    __shared__ uint32_t hist[256];
    __shared__ uint64_t s_prefix, s_mask;
    __shared__ int64_t s_krem;
    __shared__ unsigned long long s_count;
    const uint64_t *kq = keys + (int64_t)blockIdx.x * n;
    uint64_t *out = sorted + (int64_t)blockIdx.x * pow2;
    if (threadIdx.x == 0) { s_prefix = 0; s_mask = 0; s_krem = k; }
    __syncthreads();
    for (int shift = 56; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        const uint64_t prefix = s_prefix, mask = s_mask;
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
            uint64_t v = kq[i];
            if ((v & mask) == prefix) atomicAdd(&hist[(v >> shift) & 0xff], 1u);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int64_t krem = s_krem, acc = 0;
            int dgt = 0;
            for (; dgt < 256; ++dgt) {
                if (acc + (int64_t)hist[dgt] >= krem) break;
                acc += hist[dgt];
            }
            s_krem = krem - acc;
            s_prefix = prefix | ((uint64_t)dgt << shift);
            s_mask = mask | (0xffull << shift);
        }
        __syncthreads();
    }
    const uint64_t kth = s_prefix;  // exact k-th smallest key (keys are unique)
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        uint64_t v = kq[i];
        if (v <= kth) out[atomicAdd(&s_count, 1ull)] = v;
    }
    for (int64_t i = k + threadIdx.x; i < pow2; i += blockDim.x) out[i] = KEY_EMPTY;
    __syncthreads();
    for (int64_t size = 2; size <= pow2; size <<= 1) {
        for (int64_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (int64_t i = threadIdx.x; i < pow2 / 2; i += blockDim.x) {
                int64_t lo = (i / stride) * stride * 2 + (i % stride);
                int64_t hi = lo + stride;
                bool up = ((lo & size) == 0);
                uint64_t a = out[lo], b = out[hi];
                if ((a > b) == up) { out[lo] = b; out[hi] = a; }
            }
            __syncthreads();
        }
    }
}

__global__ void keys_to_output_kernel(const uint64_t *__restrict__ sorted, int64_t pow2, int64_t qc, int64_t k,
                                      int64_t q_begin, int is_hamming, int64_t *__restrict__ out_idx,
                                      void *__restrict__ out_dist) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= qc * k) return;
    const int64_t qq = t / k, j = t % k;
    uint64_t key = sorted[qq * pow2 + j];
    bool e = key == KEY_EMPTY;
    const int64_t o = (q_begin + qq) * k + j;
    out_idx[o] = e ? -1 : (int64_t)key_idx(key);
    if (is_hamming) reinterpret_cast<int64_t *>(out_dist)[o] = e ? 0 : (int64_t)key_dist(key);
    else reinterpret_cast<float *>(out_dist)[o] = e ? 0.f : __uint_as_float(key_dist(key));
}

// ── host-side launchers ───────────────────────────────────────────────────
// CTAs of the float scan per SM: three by registers, fewer by shared memory.
static int fs_occupancy(const FsGeom &g) { return (int)std::min<size_t>(3, (size_t)227 * 1024 / (g.smem + 1024)); }

// Of 1 .. hi slices the fewest whose last wave of `slots` CTAs is (nearly) fullest.
static int64_t fullest_slices(int64_t n_groups, int64_t slots, int64_t hi) {
    int64_t slices = 1;
    double best = -1.0;
    for (int64_t s = 1; s <= hi; ++s) {
        const int64_t units = n_groups * s;
        const double eff = (double)units / (double)(ceil_div(units, slots) * slots);
        if (eff > best + 0.02) {
            best = eff;
            slices = s;
        }
    }
    return slices;
}

// Slices of `stages` stages of `rows` rows for the float scan with k <= 64, at most hi: the
// fewest whose time is within 3 % of the least.  In rows, a unit takes its own and what
// starting its lists anew costs (about 5,000 coordinates' work).  Units that fit the GPU
// together take 0.63, 0.82 or all of a full wave's time, with one, two or three of them per
// SM; more of them go as slots become free, with a third of a wave left over at the end.
// Scan alone in us, by slices: 2,318 x 32 rows, 8,145 queries 1: 150, 2: 149, 4: 165, 8: 190;
// 20,000 x 8, 7,500 queries 1: 439, 2: 411, 4: 444, 8: 529; 6,592 x 12, 725 queries 3: 49, 7: 36,
// 9: 34, 13: 46.
struct SlicePlan {
    int64_t slices;
    double time;
};
static SlicePlan cheapest_slices(int64_t stages, int rows, int d, int64_t n_groups, int64_t slots) {
    const int64_t hi = std::min<int64_t>(stages, std::max<int64_t>(1, ceil_div(2 * slots, n_groups)));
    const int64_t sms = dev_info().num_sms;
    const double occ = (double)slots / (double)sms, anew = 5000.0 / std::max(d, 4);
    auto time = [&](int64_t t) {  // of slices of t stages
        const int64_t units = n_groups * ceil_div(stages, t);
        const double waves = units <= slots
                                 ? 0.45 + 0.55 * (double)ceil_div(units, sms) / occ
                                 : std::min((double)ceil_div(units, slots), (double)units / (double)slots + 0.35);
        return waves * ((double)(t * rows) + anew);
    };
    // the stages of a slice fall as the slices grow: every value once
    double least = 0.0;
    for (int64_t s = 1; s <= hi;) {
        const int64_t t = ceil_div(stages, s);
        const double c = time(t);
        if (s == 1 || c < least) least = c;
        if (t == 1) break;
        s = ceil_div(stages, t - 1);
    }
    for (int64_t s = 1;;) {
        const int64_t t = ceil_div(stages, s);
        if (time(t) <= 1.03 * least) return {ceil_div(stages, t), time(t)};
        s = ceil_div(stages, t - 1);
    }
}

void flat_plan(FlatScanArgs &a) {
    const DevInfo &di = dev_info();
    if (a.metric == M_HAMMING) {
        const size_t per_warp = (size_t)8 * a.stride4 * 16;
        int warps = 4;
        while (warps > 1 && per_warp * warps > 200 * 1024) warps >>= 1;
        a.warps = warps;
        const int64_t n_groups = ceil_div(a.nq, (int64_t)warps * 8);
        // slices of at least 128 rows, about 16 CTAs per SM over the launch
        const int64_t max_slices = std::max<int64_t>(1, a.n / 128);
        const int64_t slices = std::min<int64_t>(std::max<int64_t>(1, ceil_div(16LL * di.num_sms, n_groups)), max_slices);
        a.slice_rows = round_up(ceil_div(a.n, slices), 32);
        a.n_slices = (int)ceil_div(a.n, a.slice_rows);
        a.n_groups = (int)n_groups;
        return;
    }
    const FsGeom g = fs_geom(a.n, a.nq, a.k, a.stride4);
    const int64_t n_groups = ceil_div(a.nq, (int64_t)g.wq * g.qw);
    // up to about two waves of resident CTAs; k > 64: the slice count whose last wave is
    // fullest, the fewest slices on a tie, since every slice starts its lists empty
    const int64_t slots = (int64_t)std::max(1, fs_occupancy(g)) * di.num_sms;
    const int64_t max_slices = std::max<int64_t>(1, ceil_div(a.n, g.rows));
    int64_t slices;
    a.wave_queries = 0;
    if (a.k <= 64) {
        const SlicePlan p = cheapest_slices(max_slices, g.rows, a.d, n_groups, slots);
        slices = p.slices;
        // a batch of more than a wave and less than two: the whole wave first, the rest in
        // slices of its own, where that is worth the launches (about 8 us, 6,700 coordinates a
        // unit).  3,000 x 32 rows, 9,000 queries: 326 us a search in one piece, 306 so; 5,000 x
        // 32, 7,400: 420 and 362.
        if (n_groups > slots && n_groups < 2 * slots &&
            cheapest_slices(max_slices, g.rows, a.d, slots, slots).time +
                    cheapest_slices(max_slices, g.rows, a.d, n_groups - slots, slots).time + 6700.0 / a.d <
                0.95 * p.time)
            a.wave_queries = slots * g.wq * g.qw;
    } else {
        slices = fullest_slices(n_groups, slots,
                                std::min<int64_t>(max_slices, std::max<int64_t>(1, ceil_div(2 * slots, n_groups))));
    }
    if (n_groups * max_slices <= slots) slices = max_slices;  // one stage each
    a.slice_rows = round_up(ceil_div(a.n, slices), g.rows);
    a.n_slices = (int)ceil_div(a.n, a.slice_rows);
    a.n_groups = (int)n_groups;
    a.list_keys = (int64_t)a.n_slices * g.wr * a.k;
    a.units = (int64_t)a.n_slices * n_groups;
    a.gbuf_keys = g.cap == LIST_CAP_L ? a.units * FS_WARPS * g.qw * LIST_CAP_L : 0;
}

// Scratch: Hamming, the slices' partial lists; float, the queries' counters
// (first), candidates and, for k > 64, the scan's buffers.
size_t flat_part_bytes(const FlatScanArgs &a) {
    if (a.metric == M_HAMMING) return (size_t)a.nq * a.n_slices * a.k * sizeof(uint64_t);
    return (size_t)round_up(a.nq * 4, 256) + (size_t)(a.nq * a.list_keys + a.gbuf_keys) * sizeof(uint64_t);
}

// Rows whose queries fit the scan.  (Float: the widths accepted are those of a
// stage ring of 32-row stages of up to 256 floats beside 1, 2 or 4 queries per
// warp; what the scan itself needs is less.)
int flat_smem_ok(const FlatScanArgs &a) {
    if (a.metric == M_HAMMING) return (size_t)a.warps * 8 * a.stride4 * 16 <= (size_t)dev_info().max_smem_optin;
    const int qw = (a.k <= 32 && a.nq <= 4) ? 1 : (a.k <= 32 && a.nq <= 8) ? 2 : 4;
    const size_t per_warp = (size_t)qw * a.stride4 * 16;
    int warps = (int)std::min<int64_t>(4, std::max<int64_t>(1, ceil_div(a.nq, (int64_t)qw)));
    while (warps > 1 && per_warp * warps > 200 * 1024) warps >>= 1;
    const int nbx = (a.stride4 * 4 + FS_BOX - 1) / FS_BOX;
    const size_t stage = nbx <= 2 ? (size_t)nbx * 128 * std::min(a.stride4 * 4, FS_BOX) * 4
                                  : (size_t)std::min(nbx, 8) * 32 * FS_BOX * 4;
    return per_warp * warps + 1024 + 3 * stage + 24 <= (size_t)dev_info().max_smem_optin &&
           fs_geom(a.n, a.nq, a.k, a.stride4).smem <= (size_t)dev_info().max_smem_optin;
}

static int hamming_launch(const FlatScanArgs &a, uint64_t *part, cudaStream_t st) {
    const int units = a.n_groups * a.n_slices, threads = a.warps * 32;
    const size_t smem = (size_t)a.warps * 8 * a.stride4 * 16;
    auto go = [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        timing_begin(st, "hamming_scan_kernel");
        auto kern = hamming_scan_kernel<8, R>;
        if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        kern<<<units, threads, smem, st>>>(reinterpret_cast<const uint4 *>(a.db), a.n, a.stride4,
                                           reinterpret_cast<const uint4 *>(a.q), a.nq, a.k, a.n_slices, a.slice_rows,
                                           a.n_groups, part);
        timing_end(st);
        // a batch of up to two queries per SM over many slices: a block per query
        if (R == 1 && a.nq > 0 && a.nq <= 2 * dev_info().num_sms && a.n_slices >= 2 * MERGE_WARPS) {
            flat_merge_split_kernel<<<(unsigned)a.nq, MERGE_WARPS * 32, 0, st>>>(
                part, a.n_slices, a.k, a.out_idx, reinterpret_cast<int64_t *>(a.out_dist));
            return;
        }
        const int qpb = 4;  // queries (warps) per merge block
        flat_merge_kernel<R><<<(unsigned)ceil_div(a.nq, qpb), qpb * 32, 0, st>>>(
            part, a.n_slices, a.k, a.nq, a.out_idx, reinterpret_cast<int64_t *>(a.out_dist));
    };
    if (a.k <= 32) go(std::integral_constant<int, 1>());
    else if (a.k <= 64) go(std::integral_constant<int, 2>());
    else if (a.k <= 128) go(std::integral_constant<int, 4>());
    else go(std::integral_constant<int, 8>());
    return GN_OK;
}

template <typename Dist>
static void finish_launch(const uint64_t *cand, const int *qcount, int64_t list_keys, int64_t nq, int k,
                          int64_t *out_idx, Dist *out_dist, int64_t *out_cnt, const int *only_if, const int *err,
                          int *status, cudaStream_t st) {
    auto finish = [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        if (nq <= dev_info().num_sms && R <= 2)
            flat_finish_kernel<24, R><<<(unsigned)nq, 768, 0, st>>>(cand, qcount, list_keys, k, out_idx, out_dist,
                                                                  out_cnt, only_if, err, status);
        else if (nq <= 4 * dev_info().num_sms)
            flat_finish_kernel<8, R><<<(unsigned)nq, 256, 0, st>>>(cand, qcount, list_keys, k, out_idx, out_dist,
                                                                  out_cnt, only_if, err, status);
        else
            flat_finish_kernel<1, R><<<(unsigned)nq, 32, 0, st>>>(cand, qcount, list_keys, k, out_idx, out_dist,
                                                                  out_cnt, only_if, err, status);
    };
    if (k <= 32) finish(std::integral_constant<int, 1>());
    else if (k <= 64) finish(std::integral_constant<int, 2>());
    else if (k <= 128) finish(std::integral_constant<int, 4>());
    else finish(std::integral_constant<int, 8>());
}

int candidates_finish(const uint64_t *cand, const int *qcount, int64_t list_keys, int64_t nq, int k, int64_t *out_idx,
                      float *out_dist, int64_t *out_cnt, const int *only_if, cudaStream_t st, const int *err,
                      int *status) {
    finish_launch(cand, qcount, list_keys, nq, k, out_idx, out_dist, out_cnt, only_if, err, status, st);
    return GN_OK;
}

static int float_launch(const FlatScanArgs &a, uint64_t *part, cudaStream_t st) {
    if (!a.err) return fail(GN_ERR_INVALID, "float scan: no error word");
    const FsGeom g = fs_geom(a.n, a.nq, a.k, a.stride4);
    // the rows as a TMA tensor: n rows x dp floats, boxes of 32 floats x the stage's rows, 128-byte swizzle
    CUtensorMap tm;
    GN_TRY(tmap_encode_2d(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.db, (uint64_t)a.stride4 * 4, (uint64_t)a.n,
                          (uint64_t)a.stride4 * 16, (uint32_t)g.bw, (uint32_t)g.rows,
                          g.bw == FS_BOX ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE));
    FsArgs f;
    f.n = a.n;
    f.nq = a.nq;
    f.slice_rows = a.slice_rows;
    f.list_keys = a.list_keys;
    f.d = a.d;
    f.dp4 = a.stride4;
    f.k = a.k;
    f.n_slices = a.n_slices;
    f.n_groups = a.n_groups;
    f.wq = g.wq;
    f.wr = g.wr;
    f.nbx = g.nbx;
    f.bw = g.bw;
    f.rows = g.rows;
    f.cb = g.cb;
    f.nchunk = g.nchunk;
    f.cap = g.cap;
    f.most = g.most;
    f.q = reinterpret_cast<const float *>(a.q);
    f.qcount = reinterpret_cast<int *>(part);
    f.cand = part + round_up(a.nq * 4, 256) / 8;
    f.gbuf = f.cand + a.nq * a.list_keys;
    f.err = a.err;
    f.only_if = a.only_if;
    GN_CUDA_TRY(cudaMemsetAsync(f.qcount, 0, (size_t)a.nq * 4, st));
    if (!a.only_if) timing_begin(st, "float_scan_kernel");
    auto go = [&](auto MC) -> int {
        constexpr int M = decltype(MC)::value;
        auto launch = [&](auto kern) -> int {
            if (g.smem > 48 * 1024)
                GN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
            kern<<<(unsigned)a.units, FS_THREADS, g.smem, st>>>(tm, f);
            return GN_OK;
        };
        const bool one = g.nchunk == 1;
        if (g.rpt == 2) return one ? launch(float_scan_kernel<M, 4, 2, true>) : launch(float_scan_kernel<M, 4, 2, false>);
        if (g.qw == 4) return one ? launch(float_scan_kernel<M, 4, 1, true>) : launch(float_scan_kernel<M, 4, 1, false>);
        if (g.qw == 2) return one ? launch(float_scan_kernel<M, 2, 1, true>) : launch(float_scan_kernel<M, 2, 1, false>);
        return one ? launch(float_scan_kernel<M, 1, 1, true>) : launch(float_scan_kernel<M, 1, 1, false>);
    };
    GN_TRY(a.metric == M_L2   ? go(std::integral_constant<int, M_L2>())
           : a.metric == M_L1 ? go(std::integral_constant<int, M_L1>())
                              : go(std::integral_constant<int, M_LINF>()));
    if (!a.only_if) timing_end(st);
    return candidates_finish(f.cand, f.qcount, a.list_keys, a.nq, a.k, a.out_idx, reinterpret_cast<float *>(a.out_dist),
                             nullptr, a.only_if, st, a.err, a.status);
}

// Launch shape of hamming_append_kernel: queries per warp and warps across queries (no
// more than the batch has use for; buffers of k > 64 are 4 KB), rows per lane (more loads
// in flight where one query shares them), bytes of shared memory.
struct HamGeom {
    int qw, wq, rpt;
    size_t smem;
};
static HamGeom ham_geom(int64_t nq, int k, int w4) {
    HamGeom g;
    g.qw = nq <= 1 ? 1 : nq <= 8 || k > 64 ? 2 : 4;
    g.wq = nq <= 2 ? 1 : nq <= 4 ? 2 : 4;
    auto bytes = [&]() { return (size_t)g.qw * ((size_t)g.wq * w4 * 16 + 4 * (size_t)list_cap(k) * 8); };
    while (g.wq > 1 && bytes() > 100 * 1024) g.wq >>= 1;
    while (g.qw > 1 && bytes() > 100 * 1024) g.qw >>= 1;
    g.rpt = g.qw == 1 ? 4 : 2;
    g.smem = bytes();
    return g;
}

void ham_plan(FlatScanArgs &a) {
    const HamGeom g = ham_geom(a.nq, a.k, a.stride4);
    const int64_t n_groups = ceil_div(a.nq, (int64_t)g.qw * g.wq), unit = 32 * g.rpt * (4 / g.wq);
    const int64_t slots = std::max<int64_t>(1, std::min<int64_t>(HAM_CTAS, (int64_t)(227 * 1024 / (g.smem + 1024)))) *
                          dev_info().num_sms;
    const int64_t max_slices = std::max<int64_t>(1, ceil_div(a.n, unit));
    // two waves fill the last one better; one where slices would be short, since every
    // slice starts its lists empty (5,266 rows, 560 queries: 106 us a search with 128-row
    // slices, 102 with one wave; 1M rows, 100 queries: 517 us with two waves, 547 with one)
    const int64_t waves = a.n * n_groups >= 2048 * 2 * slots ? 2 : 1;
    const int64_t hi = std::min<int64_t>(max_slices, std::max<int64_t>(1, ceil_div(waves * slots, n_groups)));
    a.slice_rows = round_up(ceil_div(a.n, fullest_slices(n_groups, slots, hi)), unit);
    a.n_slices = (int)ceil_div(a.n, a.slice_rows);
    a.n_groups = (int)n_groups;
    a.list_keys = (int64_t)a.n_slices * (4 / g.wq) * a.k;
}

// Scratch of ham_launch: the queries' counters and bounds, then their candidates.
size_t ham_part_bytes(const FlatScanArgs &a) {
    return (size_t)round_up(a.nq * 8, 256) + (size_t)(a.nq * a.list_keys) * sizeof(uint64_t);
}

int ham_launch(const FlatScanArgs &a, uint64_t *part, cudaStream_t st) {
    const HamGeom g = ham_geom(a.nq, a.k, a.stride4);
    int *qcount = reinterpret_cast<int *>(part);
    uint64_t *cand = part + round_up(a.nq * 8, 256) / 8;
    GN_CUDA_TRY(cudaMemsetAsync(qcount, 0, (size_t)a.nq * 8, st));
    timing_begin(st, "hamming_append_kernel");
    auto launch = [&](auto kern) -> int {
        if (g.smem > 48 * 1024)
            GN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
        kern<<<(unsigned)((int64_t)a.n_groups * a.n_slices), 128, g.smem, st>>>(
            reinterpret_cast<const uint4 *>(a.db), a.n, a.stride4, reinterpret_cast<const uint4 *>(a.q), a.nq, a.k,
            list_cap(a.k), list_most(a.k), g.wq, a.slice_rows, a.n_groups, cand, a.list_keys, qcount,
            reinterpret_cast<uint32_t *>(qcount + a.nq));
        return GN_OK;
    };
    GN_TRY(g.qw == 4   ? launch(hamming_append_kernel<4, 2>)
           : g.qw == 2 ? launch(hamming_append_kernel<2, 2>)
                       : launch(hamming_append_kernel<1, 4>));
    timing_end(st);
    finish_launch<int64_t>(cand, qcount, a.list_keys, a.nq, a.k, a.out_idx, reinterpret_cast<int64_t *>(a.out_dist),
                           nullptr, nullptr, nullptr, nullptr, st);
    return GN_OK;
}

// Hamming searches that keep ordered lists (flat_plan, flat_launch) rather than appended
// candidates (ham_plan, ham_launch).  Whole searches in us, ordered / appended:
//   k > 64 with many pairs to count: two queries a warp, all that the larger buffers leave
//   room for, count slower than eight, the more so where rows are long, while the lists cost
//   the same whatever the rows.  100k x 115 bytes, k 65: 1,000 queries 3357 / 1619, 5,000
//   7393 / 8683, 14,000 15112 / 21181; k 100: 4268 / 1617, 9005 / 8705, 17105 / 21198; 500k x 64, 5,000
//   queries, k 65: 13423 / 14312; k 200 there: 43550 / 14584;
//   a handful of rows, or a few hundred for thousands of queries: little to leave out, and a
//   launch less.  120 x 64, 18,000 queries, k 4: 133 / 158; 5 x 64, 2,000: 49 / 61 (k 20 over 120
//   rows, 18,000 queries: 163 / 165);
//   rows of so few bits that most distances are tied: 15,000 x 1, 90 queries, k 4: 64 / 77.
bool ham_ordered(const FlatScanArgs &a) {
    if (a.k > 64) {
        const double work = (double)a.nq * (double)a.n * (double)(4 * a.stride4);
        return work >= (a.stride4 > 4 ? 1.2e10 : 3.5e10) * (a.k / 65.0) * (a.k > 128 ? 3.0 : 1.0);
    }
    if (a.k > 8) return false;
    const bool tied = a.d <= 2 && a.n >= (int64_t)2 << (8 * a.d);
    return a.n <= 16 || (a.n <= 512 && a.nq >= 6000) || (tied && a.nq >= 24);
}

// Launch the k <= 256 path.  part: flat_part_bytes(a) scratch.
int flat_launch(const FlatScanArgs &a, uint64_t *part, cudaStream_t st) {
    return a.metric == M_HAMMING ? hamming_launch(a, part, st) : float_launch(a, part, st);
}

int64_t next_pow2(int64_t v) {
    int64_t p = 1;
    while (p < v) p <<= 1;
    return p;
}

// Large-k path for one chunk of queries [q_begin, q_begin + qc).
// keys: qc*n scratch; sorted: qc*next_pow2(k) scratch.
void flat_large_k_launch(const FlatScanArgs &a, int64_t q_begin, int64_t qc, uint64_t *keys, uint64_t *sorted,
                         cudaStream_t st) {
    const int64_t total = qc * a.n;
    const unsigned blocks = (unsigned)ceil_div(total, 256);
    switch (a.metric) {
    case M_HAMMING: flat_keys_kernel<M_HAMMING><<<blocks, 256, 0, st>>>(a.db, a.n, a.d, a.stride4, a.q, q_begin, qc, keys); break;
    case M_L2: flat_keys_kernel<M_L2><<<blocks, 256, 0, st>>>(a.db, a.n, a.d, a.stride4, a.q, q_begin, qc, keys); break;
    case M_L1: flat_keys_kernel<M_L1><<<blocks, 256, 0, st>>>(a.db, a.n, a.d, a.stride4, a.q, q_begin, qc, keys); break;
    default: flat_keys_kernel<M_LINF><<<blocks, 256, 0, st>>>(a.db, a.n, a.d, a.stride4, a.q, q_begin, qc, keys); break;
    }
    const int64_t kk = std::min<int64_t>(a.k, a.n);
    const int64_t p2 = next_pow2(a.k);
    radix_select_sort_kernel<<<(unsigned)qc, 1024, 0, st>>>(keys, a.n, kk, p2, sorted);
    keys_to_output_kernel<<<(unsigned)ceil_div(qc * a.k, 256), 256, 0, st>>>(sorted, p2, qc, a.k, q_begin,
                                                                              a.metric == M_HAMMING, a.out_idx,
                                                                              a.out_dist);
}

}  // namespace gn

namespace gn {

// Loads every kernel the Hamming warp-select path can launch (the scan and
// the merge, for each list width).  With lazy module loading (the default
// since CUDA 12.2) a kernel's module is loaded, and its device memory
// allocated, at its first launch; querying the kernel's attributes loads it
// ahead of that.  Cheap once loaded.
int flat_preload_hamming() {
    cudaFuncAttributes fa;
    const void *fns[] = {(const void *)hamming_scan_kernel<8, 1>, (const void *)hamming_scan_kernel<8, 2>,
                         (const void *)hamming_scan_kernel<8, 4>, (const void *)hamming_scan_kernel<8, 8>,
                         (const void *)flat_merge_kernel<1>,      (const void *)flat_merge_kernel<2>,
                         (const void *)flat_merge_kernel<4>,      (const void *)flat_merge_kernel<8>,
                         (const void *)flat_merge_split_kernel};
    for (const void *f : fns) GN_CUDA_TRY(cudaFuncGetAttributes(&fa, f));
    return GN_OK;
}

}  // namespace gn
