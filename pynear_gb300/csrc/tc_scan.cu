// tc_scan.cu — tensor-core candidate scans: a tcgen05 GEMM with a fused
// per-query top-S epilogue, and the exact FP32 re-rank that follows it.
//
// Used by the flat L2 shortlist (BF16, or FP8 E4M3 with one FP32 scale per
// row; rows scored as |x|^2 - 2 q.x) and by large batches of the exact Hamming
// scan (bits as E4M3 +1 / -1: the inner product of two rows is nbits - 2 h,
// exact in FP32, so the "shortlist" is the answer).
//
// One persistent CTA per SM walks work units.  A unit is one or two M = 128 tiles
// of queries ("A" rows) against a chunk of the database ("B" rows, taken 256 at
// a time), all K-major; a pipeline stage holds 128 bytes of K per row.
//   warp 0     TMA producer: the unit's queries once (where their K fits shared
//              memory: "resident"), then 256-row, 128-byte K slices of the
//              database into a ring (otherwise a query slice rides along), and
//              the rows' norms into a ring of their own (whose slots the epilogue
//              gives back behind a fence: mbar_release_warp);
//   warp 1     allocates 512 TMEM columns, one thread issues tcgen05.mma
//              (M=128, N=256) into one of two 256-column accumulators, query
//              tile by query tile for each database tile;
//   warps 2-17 epilogue: TMEM lane quadrant x column quarter; thread = query.
//              tcgen05.ld of 32 columns at a time; a block's smallest score
//              against the query's threshold ends most blocks.
//              Passing (score, row) pairs are appended to the query's buffer
//              in global memory (a plain store, no list is kept in order);
//              only a buffer that fills is sorted, by its warp, down to the S
//              best, whose last is the new threshold.
// At the end of a unit each thread appends its buffer (at most the S best of it)
// to the query's candidate list, whose length the re-rank reads.
//
// What makes passing scores rare is the bound that every unit starts from.
// With a warp's 32 lanes being 32 queries, a block of 32 x 32 scores is only
// cheap when none of 1,024 passes.  So a pilot launch of the same pipeline first
// scores every 8th row or so (all rows of a small database; none where the buffers
// hold them all) and keeps, per query, only the minima of groups
// of rows (32 per unit, one per column of a block: no insertion, no branch).
// The S-th smallest minimum over at least S groups is a score that at least S
// rows reach, hence an upper bound of the query's S-th best score, and close
// to the sample's own S-th best (1/8 of the rows: about 320 rows of the
// database pass instead of 1,600 per unit from empty lists).  Rows at the bound pass,
// so the S best (score, row) keys are the same as without it.
//
// Two query tiles per unit (where a whole database tile fits the ring, K of at
// most 256 bytes) because one, with its queries streamed next to each database
// slice, read 30 GB through L2 for 1M x 128 and 10k queries and kept to 1.0 of
// 1.93 PFLOP/s without any epilogue work; resident queries used twice read 10 GB.
// N = 256 rather than 128 because the issuing thread's waits and commits, about
// 300 cycles each, stand beside every 128 bytes of K.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include <algorithm>

#include "distance.cuh"
#include "f32x2.cuh"
#include "gemm_topk.cuh"
#include "index.cuh"
#include "kmeans.cuh"
#include "select.cuh"
#include "tc_scan.cuh"
#include "tc_sm100.cuh"
#include "tmap.cuh"
#include "timing.cuh"
#include "topk.cuh"

namespace gn {

constexpr int TC_M = 128, TC_N = 256;   // queries per MMA tile, database rows per tile
constexpr int TC_BK = 64;               // BF16 elements per 128-byte K slice
constexpr int TC_BK8 = 128;             // FP8 elements per 128-byte K slice
constexpr int TC_ASLICE = TC_M * 128;   // bytes of a K slice of a query tile
constexpr int TC_BSLICE = TC_N * 128;   // ... of a database tile
constexpr int TC_NEPI = 16;             // epilogue warps: TMEM lane quadrant x column quarter (eight warps of
                                        // two quarters each were bound by their own latency: 440 cycles a block)
constexpr int TC_COLS = TC_N / (TC_NEPI / 4);  // columns of a tile per epilogue warp
constexpr int TC_THREADS = 64 + 32 * TC_NEPI;
constexpr int TC_MAX_STAGES = 6;
constexpr int TC_NR = 4;                // tiles of row norms (and scales) in flight
constexpr int64_t TC_EXACT_MIN = 4096;  // rows from which exact Hamming and L2 searches come here
constexpr int64_t TC_QBLOCK = 65536;    // queries scanned at a time (bounds the scratch) ...
constexpr int64_t L2TC_QBLOCK = 8192;   // ... and by the exact L2 search, whose candidate lists are longer
constexpr int TC_CAP = 128;             // entries of a buffer (S <= 64, and a block adds up to 32)

// Shared memory: [queries, resident: qt x nk slices][ring][norms, scales of TC_NR tiles][barriers].
struct TcGeom {
    int nk, qt, resident, stages;
    size_t stage_bytes, smem;
};
static TcGeom tc_geom(int nk, bool pilot) {
    constexpr size_t fixed = 1024 + (size_t)TC_NR * TC_N * 4 * 2 + 256;  // alignment, norms and scales, barriers
    constexpr size_t room = 227 * 1024 - fixed;
    TcGeom g;
    g.nk = nk;
    g.qt = nk <= 2 && !pilot ? 2 : 1;  // the pilot keeps its minima in registers: one query tile
    g.resident = nk <= 6;
    g.stage_bytes = g.resident ? TC_BSLICE : TC_BSLICE + TC_ASLICE;
    const size_t a = g.resident ? (size_t)nk * g.qt * TC_ASLICE : 0;
    g.stages = (int)std::min<size_t>(TC_MAX_STAGES, (room - a) / g.stage_bytes);
    g.smem = fixed + a + (size_t)g.stages * g.stage_bytes;
    return g;
}

// A buffer entry is (score bits, row); keys order by (score, row).  (Signs: the
// score is -(inner product) = 2 h - nbits, and the candidate list gets (h, row).)
__device__ __forceinline__ uint64_t tc_entry_key(const uint2 *buf, int i, int cnt) {
    if (i >= cnt) return KEY_EMPTY;
    const uint2 e = buf[i];
    return make_key(f2ord(__uint_as_float(e.x)), e.y);
}

// The warp sorts the first cnt entries of buf (cnt <= 32 R), writes the S best
// back, and returns the S-th key (KEY_EMPTY if there are fewer).
template <int R>
__device__ __forceinline__ uint64_t tc_compact(uint2 *buf, int cnt, int S) {
    const int lane = threadIdx.x & 31;
    uint64_t v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = tc_entry_key(buf, r * 32 + lane, cnt);
    warp_sort<R>(v);
    __syncwarp();
    uint64_t last = KEY_EMPTY;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = r * 32 + lane;
        if (p < S && v[r] != KEY_EMPTY) buf[p] = make_uint2(__float_as_uint(ord2f(key_dist(v[r]))), key_idx(v[r]));
        if (r == (S - 1) / 32) last = __shfl_sync(0xffffffffu, v[r], (S - 1) & 31);
    }
    __syncwarp();
    return last;
}

__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// MODE: operand form.  PILOT: group minima of the sampled tiles instead of lists.
// QT: query tiles per unit.  Unit u is (chunk u / nqp of the tiles, queries 128 QT (u % nqp) ..): chunk-major,
// so that the CTAs running together scan the same chunk and L2 serves it.
template <int MODE, bool PILOT, int QT>
__global__ void __launch_bounds__(TC_THREADS, 1)
    tc_topk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, TcScanArgs a) {
    static_assert(!PILOT || QT == 1, "the pilot's minima are one query tile's");
    constexpr int UQ = TC_M * QT;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int nk = a.nk, ST = a.stages;
    const bool res = QT == 2 || a.resident != 0;
    const uint32_t stage_bytes = res ? TC_BSLICE : TC_BSLICE + TC_ASLICE;
    uint8_t *sA = smem;  // resident queries: slice (qt, kb) at (qt * nk + kb) * TC_ASLICE
    uint8_t *ring = smem + (res ? (size_t)nk * QT * TC_ASLICE : 0);  // stage: database slice [, query slice]
    float *snorm = reinterpret_cast<float *>(ring + (size_t)ST * stage_bytes);  // [TC_NR][TC_N] norms, then scales
    float *sscale = snorm + TC_NR * TC_N;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sscale + TC_NR * TC_N);
    uint64_t *full = bars, *empty = bars + TC_MAX_STAGES, *nfull = bars + 2 * TC_MAX_STAGES, *nempty = nfull + TC_NR,
             *accfull = nempty + TC_NR, *accempty = accfull + 2, *afull = accfull + 4, *aempty = accfull + 5,
             *drain = accfull + 6;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accfull + 7);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *verr = a.err;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accfull + b, 1);
            mbar_init(accempty + b, TC_NEPI);
        }
        for (int b = 0; b < TC_NR; ++b) {
            mbar_init(nfull + b, 1);
            mbar_init(nempty + b, TC_NEPI);
        }
        mbar_init(afull, 1);
        mbar_init(aempty, 1);
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    const int64_t nqp = (a.nq + UQ - 1) / UQ;
    const int64_t n_units = nqp * a.nchunks;
    auto unit = [&](int64_t u, int64_t &q0, int &na, int64_t &t0, int64_t &t1) {
        const int64_t c = u / nqp;
        q0 = (u % nqp) * UQ;
        na = (int)min((int64_t)UQ, a.nq - q0);
        t0 = a.ntiles * c / a.nchunks;
        t1 = a.ntiles * (c + 1) / a.nchunks;
        return c;
    };

    if (warp == 0) {
        // ── TMA producer ──
        if (lane == 0) {
            uint32_t it = 0, aloads = 0, nloads = 0;  // copies issued: slices, units' queries, tiles' norms
            int sl = 0;
            uint32_t ph = 1;  // parity of the ring pass before this one: slots start free
            bool ok = true;
            for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
                int64_t q0, t0, t1;
                int na;
                unit(u, q0, na, t0, t1);
                const int nqt = QT == 2 && na > TC_M ? 2 : 1;
                if (res) {  // the unit's queries, once the previous unit's MMAs have read theirs
                    if (!mbar_wait(aempty, (aloads & 1) ^ 1, verr)) { ok = false; break; }
                    mbar_expect_tx(afull, (uint32_t)(nqt * nk) * TC_ASLICE);
                    for (int qt = 0; qt < nqt; ++qt)
                        for (int kb = 0; kb < nk; ++kb)
                            tma_load_2d(sA + (size_t)(qt * nk + kb) * TC_ASLICE, &tmA, kb * a.kblk,
                                        (int)(q0 + qt * TC_M), afull);
                    ++aloads;
                }
                for (int64_t t = t0; t < t1 && ok; ++t) {
                    const int n0 = (int)(t * TC_N);
                    for (int kb = 0; kb < nk; ++kb, ++it) {
                        if (!mbar_wait(empty + sl, ph, verr)) { ok = false; break; }
                        uint8_t *sb = ring + (size_t)sl * stage_bytes;
                        mbar_expect_tx(full + sl, stage_bytes);
                        tma_load_2d(sb, &tmB, kb * a.kblk, n0, full + sl);
                        if (!res) tma_load_2d(sb + TC_BSLICE, &tmA, kb * a.kblk, (int)q0, full + sl);
                        if (++sl == ST) {
                            sl = 0;
                            ph ^= 1;
                        }
                    }
                    if (MODE != TC_SIGN && ok) {
                        const int ns = nloads % TC_NR;
                        if (!mbar_wait(nempty + ns, ((nloads / TC_NR) & 1) ^ 1, verr)) { ok = false; break; }
                        mbar_expect_tx(nfull + ns, TC_N * 4 * (MODE == TC_FP8 ? 2 : 1));
                        bulk_load(snorm + ns * TC_N, a.bnorm + n0, TC_N * 4, nfull + ns);
                        if (MODE == TC_FP8) bulk_load(sscale + ns * TC_N, a.bscale + n0, TC_N * 4, nfull + ns);
                        ++nloads;
                    }
                }
            }
            if (!ok) {  // let the copies in flight land (bounded) before the CTA ends
                auto settle = [&](uint64_t *bar, uint32_t parity) {
                    const long long c0 = clock64();
                    while (!mbar_try_wait(bar, parity) && clock64() - c0 < 400000) {
                    }
                };
                for (uint32_t x = it > (uint32_t)ST ? it - ST : 0; x < it; ++x) settle(full + x % ST, (x / ST) & 1);
                for (uint32_t x = nloads > TC_NR ? nloads - TC_NR : 0; x < nloads; ++x)
                    settle(nfull + x % TC_NR, (x / TC_NR) & 1);
                if (aloads) settle(afull, (aloads - 1) & 1);
            }
        }
    } else if (warp == 1) {
        // ── MMA issuer ──
        if (lane == 0) {
            constexpr uint32_t idesc = MODE == TC_BF16 ? idesc_bf16_f32(TC_M, TC_N) : idesc_e4m3_f32(TC_M, TC_N);
            const uint64_t ring_desc = sdesc_sw128(smem_u32(ring)), a_desc = sdesc_sw128(smem_u32(sA));
            const uint32_t stage16 = stage_bytes >> 4;  // descriptor addresses count 16-byte units
            uint32_t vt = 0, un = 0, ph = 0, sl = 0;    // vt: accumulators filled so far
            bool ok = true;
            for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++un) {
                int64_t q0, t0, t1;
                int na;
                unit(u, q0, na, t0, t1);
                const int nqt = QT == 2 && na > TC_M ? 2 : 1;
                if (res && !mbar_wait(afull, un & 1, verr)) { ok = false; break; }
                const int tiles = (int)(t1 - t0);
                for (int t = 0; t < tiles && ok; ++t) {
                    for (int qt = 0; qt < nqt && ok; ++qt, ++vt) {
                        const uint32_t b = vt & 1;
                        if (!mbar_wait(accempty + b, ((vt >> 1) & 1) ^ 1, verr)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t dt = tmem + b * TC_N;
                        uint32_t s = sl, sph = ph;  // each query tile takes the tile's slices anew
                        for (int kb = 0; kb < nk; ++kb) {
                            if (qt == 0) {
                                if (!mbar_wait(full + s, sph, verr)) { ok = false; break; }
                                tc_fence_after();
                            }
                            const uint64_t db = ring_desc + s * stage16;
                            const uint64_t da = res ? a_desc + (uint32_t)(qt * nk + kb) * (TC_ASLICE >> 4)
                                                    : db + (TC_BSLICE >> 4);
                            // four MMAs of 32 bytes of K each (16 BF16 or 32 FP8 elements):
                            // the descriptors advance by 32 bytes (2 in 16-byte units)
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                if constexpr (MODE == TC_BF16)
                                    umma_bf16(dt, da + 2 * kk, db + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                                else
                                    umma_f8(dt, da + 2 * kk, db + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                            }
                            if (qt == nqt - 1) umma_commit(empty + s);
                            if (++s == (uint32_t)ST) {
                                s = 0;
                                sph ^= 1;
                            }
                        }
                        if (ok) umma_commit(accfull + b);
                        if (qt == nqt - 1) {
                            sl = s;
                            ph = sph;
                        }
                    }
                }
                if (ok && res) umma_commit(aempty);
            }
            if (!ok) {  // the MMAs issued so far end (bounded) before the CTA does
                umma_commit(drain);
                const long long c0 = clock64();
                while (!mbar_try_wait(drain, 0) && clock64() - c0 < 400000) {
                }
            }
        }
    } else {
        // ── epilogue ──
        const int quad = warp & 3, ew = warp - 2, quarter = ew >> 2;
        uint2 *const ebuf = a.cand + ((size_t)blockIdx.x * TC_NEPI + ew) * QT * 32 * TC_CAP;  // the warp's buffers
        const float inf = __int_as_float(0x7f800000);
        uint32_t tile_it = 0, vt = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            int64_t q0, t0, t1;
            int na;
            const int64_t chunk = unit(u, q0, na, t0, t1);
            const int nqt = QT == 2 && na > TC_M ? 2 : 1;
            // per query tile: scores at or below thr pass; cnt of them are in the buffer.
            // The current tile's state is thr[0], cnt[0] (the tiles take turns)
            float thr[QT], qc[QT];
            int cnt[QT];
#pragma unroll
            for (int i = 0; i < QT; ++i) {
                const int row = i * TC_M + quad * 32 + lane;  // query within the unit
                const bool live = row < na;
                thr[i] = live ? inf : __int_as_float(0x7fc00000);  // NaN: nothing passes
                cnt[i] = 0;
                if (!PILOT && live) {
                    const uint32_t g = *reinterpret_cast<volatile uint32_t *>(a.qbound + q0 + row);
                    if (g != 0xffffffffu) thr[i] = ord2f(g);
                }
                // score = |x|^2 + qc * (column factor) * acc: qc = -2 (BF16) or
                // -2 scale_q (FP8, column factor scale_x); signs: -acc
                qc[i] = -2.f;
                if (MODE == TC_FP8) qc[i] = live ? -2.f * __ldg(a.ascale + q0 + row) : 0.f;
            }
            float g[PILOT ? 32 : 1];
#pragma unroll
            for (int j = 0; j < (PILOT ? 32 : 1); ++j) g[j] = inf;

            for (int64_t t = t0; t < t1 && ok; ++t, ++tile_it) {
                const int64_t n0 = t * TC_N + quarter * TC_COLS;
                const bool tail = MODE == TC_SIGN && n0 + TC_COLS > a.n;
                const int ns = tile_it % TC_NR;
                // the tile's row norms (NaN past the last row: such scores never pass)
                const float *sn = snorm + ns * TC_N + quarter * TC_COLS, *sc = sn + TC_NR * TC_N;
#pragma unroll 1
                for (int qt = 0; qt < nqt; ++qt, ++vt) {
                    const int b = vt & 1;
                    if (!mbar_wait_warp(accfull + b, (vt >> 1) & 1, verr)) { ok = false; break; }
                    tc_fence_after();
                    if (MODE != TC_SIGN && qt == 0 && !mbar_wait_warp(nfull + ns, (tile_it / TC_NR) & 1, verr)) {
                        ok = false;
                        break;
                    }
                    uint2 *const wbuf = ebuf + (size_t)qt * 32 * TC_CAP;
                    uint2 *const buf = wbuf + (size_t)lane * TC_CAP;
                    const f32x2 qc2 = dup2(qc[0]);
                    const uint32_t tacc =
                        tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(b * TC_N + quarter * TC_COLS);
                    // v: accumulators of the warp's columns [32 c, 32 c + 32), then their scores
                    auto block = [&](float (&v)[32], int c) {
                        if (MODE == TC_SIGN) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = -v[j];
                            if (tail) {
#pragma unroll
                                for (int j = 0; j < 32; ++j)
                                    if (n0 + c * 32 + j >= a.n) v[j] = __int_as_float(0x7fc00000);
                            }
                        } else {
                            const float4 *sn4 = reinterpret_cast<const float4 *>(sn + c * 32);
                            const float4 *sc4 = reinterpret_cast<const float4 *>(sc + c * 32);
#pragma unroll
                            for (int j4 = 0; j4 < 8; ++j4) {
                                const float4 nv = sn4[j4];
                                f32x2 f01 = qc2, f23 = qc2;
                                if (MODE == TC_FP8) {
                                    const float4 sv = sc4[j4];
                                    f01 = pack2(__fmul_rn(qc[0], sv.x), __fmul_rn(qc[0], sv.y));
                                    f23 = pack2(__fmul_rn(qc[0], sv.z), __fmul_rn(qc[0], sv.w));
                                }
                                float *x = v + 4 * j4;
                                unpack2(fma2(f01, pack2(x[0], x[1]), pack2(nv.x, nv.y)), x[0], x[1]);
                                unpack2(fma2(f23, pack2(x[2], x[3]), pack2(nv.z, nv.w)), x[2], x[3]);
                            }
                        }
                        if (PILOT) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) g[PILOT ? j : 0] = fminf(g[PILOT ? j : 0], v[j]);
                            return;
                        }
                        float m[4];  // minima of eight columns each
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float *x = v + 8 * e;
                            m[e] = min3(min3(x[0], x[1], x[2]), min3(x[3], x[4], x[5]), fminf(x[6], x[7]));
                        }
                        if (!__any_sync(0xffffffffu, fminf(fminf(m[0], m[1]), fminf(m[2], m[3])) <= thr[0])) return;
                        const uint32_t col = (uint32_t)(n0 + c * 32);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if (!__any_sync(0xffffffffu, m[e] <= thr[0])) continue;
#pragma unroll
                            for (int j = 8 * e; j < 8 * e + 8; ++j)
                                if (v[j] <= thr[0]) {
                                    buf[cnt[0]] = make_uint2(__float_as_uint(v[j]), col + j);
                                    ++cnt[0];
                                }
                        }
                        unsigned fullm = __ballot_sync(0xffffffffu, cnt[0] > TC_CAP - 32);
                        if (fullm && a.overflow) *a.overflow = 1;
                        while (fullm) {  // the warp sorts a lane's buffer down to its S best
                            const int l = __ffs(fullm) - 1;
                            fullm &= fullm - 1;
                            __syncwarp();
                            const uint64_t last = tc_compact<TC_CAP / 32>(
                                wbuf + (size_t)l * TC_CAP, __shfl_sync(0xffffffffu, cnt[0], l), a.S);
                            if (lane == l) {
                                cnt[0] = a.S;
                                // later rows of the unit have higher indices: only lower scores displace the S-th
                                thr[0] = fminf(thr[0], ord2f(key_dist(last) - 1));
                            }
                        }
                    };
                    static_assert(TC_COLS == 64, "two blocks per warp and tile");
                    float acc[32];
                    tmem_ld32(tacc, acc);
                    block(acc, 0);
                    tmem_ld32(tacc + 32, acc);
                    // every column is in registers: a later tile may overwrite the accumulator
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accempty + b);
                    block(acc, 1);
                    if (MODE != TC_SIGN && qt == nqt - 1) mbar_release_warp(nempty + ns);
                    if (QT == 2 && nqt == 2) {  // the other query tile's turn
                        const float tf = thr[0], tq = qc[0];
                        const int ti = cnt[0];
                        thr[0] = thr[QT - 1];
                        qc[0] = qc[QT - 1];
                        cnt[0] = cnt[QT - 1];
                        thr[QT - 1] = tf;
                        qc[QT - 1] = tq;
                        cnt[QT - 1] = ti;
                    }
                }
            }
            if (!ok) break;
            if (PILOT) {
                if (quad * 32 + lane < na) {
                    float4 *dst = reinterpret_cast<float4 *>(
                        a.gmin + (((q0 + quad * 32 + lane) * a.nchunks + chunk) * (TC_NEPI / 4) + quarter) * 32);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        dst[j] = make_float4(g[PILOT ? 4 * j : 0], g[PILOT ? 4 * j + 1 : 0], g[PILOT ? 4 * j + 2 : 0],
                                             g[PILOT ? 4 * j + 3 : 0]);
                }
            } else {
                __syncwarp();
#pragma unroll 1
                for (int i = 0; i < nqt; ++i) {
                    const int row = i * TC_M + quad * 32 + lane;
                    int n = i == 0 ? cnt[0] : cnt[QT - 1];
                    uint2 *const wbuf = ebuf + (size_t)i * 32 * TC_CAP;
                    unsigned longm = __ballot_sync(0xffffffffu, n > a.keep);
                    if (longm && a.overflow) *a.overflow = 1;
                    while (longm) {  // only a buffer's S best can be among the query's, and more have no room
                        const int l = __ffs(longm) - 1;
                        longm &= longm - 1;
                        const uint64_t last = tc_compact<TC_CAP / 32>(wbuf + (size_t)l * TC_CAP,
                                                                      __shfl_sync(0xffffffffu, n, l), a.S);
                        if (lane == l) {
                            n = a.S;
                            // a full list bounds the query's S-th best score for later units
                            atomicMin(a.qbound + q0 + row, key_dist(last));
                        }
                    }
                    if (row < na && n > 0) {
                        const int64_t q = q0 + row;
                        uint64_t *dst = a.part + q * a.slot_keys + atomicAdd(a.qcount + q, n);
                        const uint2 *src = wbuf + (size_t)lane * TC_CAP;
#pragma unroll 4
                        for (int e = 0; e < n; ++e) {
                            const uint2 x = src[e];
                            const float sc = __uint_as_float(x.x);
                            dst[e] = make_key(MODE == TC_SIGN ? (uint32_t)((a.nbits + (int)sc) >> 1) : f2ord(sc), x.y);
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// A query's bound from the pilot's minima (m groups of 32, warp per query): the
// S-th smallest of up to 128 groups' minima (groups joined four ways beyond
// that) is reached by at least S rows.  Fewer than S groups: no bound.
// sl.q2 given: the bound is raised so that it holds for exact distances too (see
// l2_tc_search): B -> B + 2 E + rel (B + |q|^2 + E), E = sl.cross |q| max|x| +
// sl.norm max|x|^2, and *sl.overflow is set where that is not finite.
__global__ void tc_bound_kernel(const float *__restrict__ gmin, int m, int64_t nq, int S, TcSlack sl,
                                uint32_t *__restrict__ qbound) {
    const int lane = threadIdx.x & 31;
    const int64_t q = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= nq) return;
    const float *p = gmin + q * m * 32;
    const float inf = __int_as_float(0x7f800000);
    float g[4] = {inf, inf, inf, inf};
    for (int i = 0; i < m; i += 4) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (i + r < m) g[r] = fminf(g[r], p[(i + r) * 32 + lane]);
    }
    uint64_t v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = r < m ? make_key(f2ord(g[r]), (uint32_t)(r * 32 + lane)) : KEY_EMPTY;
    warp_sort<4>(v);
    uint64_t key = KEY_EMPTY;
#pragma unroll
    for (int r = 0; r < 4; ++r)
        if (r == (S - 1) / 32) key = __shfl_sync(0xffffffffu, v[r], (S - 1) & 31);
    if (lane != 0) return;
    uint32_t bound = key == KEY_EMPTY ? 0xffffffffu : key_dist(key);
    if (sl.q2 && bound != 0xffffffffu) {
        const float b = ord2f(bound), q2 = sl.q2[q], x2 = __uint_as_float(*sl.xmax2);
        // (1e-35: products that a unit may flush to zero)
        const float e = __fadd_ru(__fadd_ru(__fmul_ru(sl.cross, __fsqrt_ru(__fmul_ru(q2, x2))), __fmul_ru(sl.norm, x2)),
                                  1e-35f);
        const float d = fmaxf(0.f, __fadd_ru(__fadd_ru(b, q2), e));
        const float raised = __fadd_ru(__fadd_ru(b, __fmul_ru(2.f, e)), __fmul_ru(sl.rel, d));
        bound = raised < inf ? f2ord(raised) : 0xffffffffu;
        if (!(raised < inf)) *sl.overflow = 1;  // NaN or infinite: scores say nothing
    }
    qbound[q] = bound;
}

// ── host: tensor maps, plan and launch ────────────────────────────────────
// K-major operand rows of K elements (BF16, or FP8 stored as bytes), boxes of
// 128 bytes of K by box_rows rows, 128-byte swizzle; stride: every stride-th row.
static int make_tmap_rows(CUtensorMap *map, const void *base, int64_t rows, int64_t K, int box_rows, bool f8,
                          int stride = 1) {
    return tmap_encode_2d(map, f8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base,
                          (uint64_t)K, (uint64_t)rows, (uint64_t)K * (f8 ? 1 : 2) * stride, f8 ? TC_BK8 : TC_BK,
                          (uint32_t)box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Chunks of the nt tiles: the smallest count whose units fill whole waves of
// CTAs best, at least `lo`, chunks of at least `tiles` tiles.
static int64_t tc_chunks(int64_t nqp, int64_t nt, int64_t lo, int64_t hi, int64_t tiles) {
    const int sms = dev_info().num_sms;
    hi = std::max<int64_t>(1, std::min(hi, nt / std::max<int64_t>(1, tiles)));
    lo = std::min(lo, hi);
    int64_t best = lo;
    double eff_best = -1.0;
    for (int64_t c = lo; c <= hi; ++c) {
        const int64_t units = nqp * c;
        const double eff = (double)units / (double)(ceil_div(units, sms) * sms);
        if (eff > eff_best + 0.01) {
            eff_best = eff;
            best = c;
        }
    }
    return best;
}

// Rows, not whole tiles, are sampled: where near rows stand together in the
// database, tiles would miss most queries' neighbourhoods.
int tc_pilot_stride(int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>(8, n / 16384));
}

// Every stride-th of n values, whole tiles of them (NaN past the last).
__global__ void tc_stride_kernel(const float *__restrict__ x, int64_t n, int stride, int64_t m,
                                 float *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) out[i] = i * stride < n ? x[i * stride] : __int_as_float(0x7fc00000);
}

static size_t tc_pilot_count(int64_t n) { return (size_t)round_up(ceil_div(n, tc_pilot_stride(n)), TC_N); }

int tc_pilot_values(const float *x, int64_t n, DBuf &out, cudaStream_t st) {
    const int stride = tc_pilot_stride(n);
    const int64_t m = (int64_t)tc_pilot_count(n);
    GN_TRY(out.ensure((size_t)m * 4));
    tc_stride_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, st>>>(x, n, stride, m, out.as<float>());
    return GN_OK;
}

static int tc_slices(int mode, int K) { return K / (mode == TC_BF16 ? TC_BK : TC_BK8); }

TcPlan tc_plan(int mode, int K, int64_t nq, int64_t n, int S) {
    TcPlan p;
    const int nk = tc_slices(mode, K);
    const int64_t sms = dev_info().num_sms, nt = ceil_div(n, TC_N);
    const int64_t nqp = ceil_div(nq, TC_M * tc_geom(nk, false).qt), nqp1 = ceil_div(nq, TC_M);
    // about five units per SM at most: shorter ones sort more lists at their ends
    // than they save in the last wave
    p.nchunks = (int)tc_chunks(nqp, nt, 1, std::min<int64_t>(64, std::max<int64_t>(1, ceil_div(5 * sms, nqp))), 2);
    // pilot: every 8th row (more where that would be under 16k rows), whole tiles
    // of them.  It pays for small databases as well, where the units' buffers would
    // fill with most rows they see: 24,813 x 126 rows, 2,956 queries, S 40: 1289 us per
    // search without it, below 300 with it; 255 x 64 rows, 5,000 queries, S 32: 388 and 152.
    // (Of at most 48 rows too many pass all the same.)
    if (n > std::max(S, 48)) {
        p.pilot_stride = tc_pilot_stride(n);
        p.pilot_tiles = std::max<int64_t>(1, n / p.pilot_stride / TC_N);
        // 128 groups of minima per chunk
        p.pilot_chunks = (int)tc_chunks(nqp1, p.pilot_tiles, 1, std::max<int64_t>(1, ceil_div(4 * sms, nqp1)), 2);
    }
    // A unit hands over its S best of each buffer, or, from a single tile, all of its columns:
    // many of few rows pass, and sorting a warp's 32 buffers one after another costs more
    // than their keys (82 x 50 rows, 3,618 queries, S 48: 380 us with it, 244 without)
    p.keep = nt == 1 ? std::max(S, TC_COLS) : S;
    p.slot_keys = (int64_t)p.nchunks * (TC_NEPI / 4) * p.keep;
    return p;
}

int tc_topk_launch(const TcLaunch &a, const TcPlan &p, TcScratch &sc, cudaStream_t st) {
    const bool f8 = a.mode != TC_BF16;
    const int kblk = f8 ? TC_BK8 : TC_BK;
    if (a.K <= 0 || a.K % kblk) return fail(GN_ERR_INVALID, "tensor-core scan: K must be whole 128-byte slices");
    if (a.S < 1 || a.S > TC_CAP - 32) return fail(GN_ERR_UNSUPPORTED, "tensor-core scan: too many results per query");
    if (a.mode == TC_FP8 && (!a.ascale || !a.bscale)) return fail(GN_ERR_INVALID, "FP8 shortlist: no row scales");
    CUtensorMap ma, mb, mp;
    GN_TRY(make_tmap_rows(&ma, a.A, a.a_rows, a.K, TC_M, f8));
    GN_TRY(make_tmap_rows(&mb, a.B, a.b_rows, a.K, TC_N, f8));
    const int sms = dev_info().num_sms;
    GN_TRY(sc.qbound.ensure((size_t)a.nq * 4));
    GN_TRY(sc.cand.ensure((size_t)sms * TC_NEPI * 2 * 32 * TC_CAP * sizeof(uint2)));
    TcScanArgs s;
    s.nq = a.nq;
    s.kblk = kblk;
    s.S = a.S;
    s.keep = p.keep;
    s.nbits = a.nbits;
    s.ascale = a.ascale;
    s.part = a.part;
    s.qcount = a.qcount;
    s.slot_keys = p.slot_keys;
    s.qbound = sc.qbound.as<uint32_t>();
    s.cand = sc.cand.as<uint2>();
    s.gmin = nullptr;
    s.err = a.err;
    s.overflow = a.overflow;
    auto run = [&](auto kern, const TcGeom &g, const CUtensorMap &mb) -> int {
        s.nk = g.nk;
        s.stages = g.stages;
        s.resident = g.resident;
        GN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
        const int64_t units = ceil_div(a.nq, TC_M * g.qt) * s.nchunks;
        kern<<<(unsigned)std::min<int64_t>(sms, units), TC_THREADS, g.smem, st>>>(ma, mb, s);
        return GN_OK;
    };
    const TcGeom g = tc_geom(a.K / kblk, false);
    GN_CUDA_TRY(cudaMemsetAsync(a.qcount, 0, (size_t)a.nq * 4, st));
    if (p.pilot_chunks) {
        const TcGeom gp = tc_geom(a.K / kblk, true);
        GN_TRY(make_tmap_rows(&mp, a.B, std::max<int64_t>(a.n / p.pilot_stride, TC_N), a.K, TC_N, f8, p.pilot_stride));
        GN_TRY(sc.gmin.ensure((size_t)a.nq * p.pilot_chunks * TC_N / 2 * 4));
        s.gmin = sc.gmin.as<float>();
        s.nchunks = p.pilot_chunks;
        s.ntiles = p.pilot_tiles;
        s.n = p.pilot_tiles * TC_N;
        s.bnorm = a.pnorm;
        s.bscale = a.pscale;
        GN_TRY(a.mode == TC_BF16  ? run(tc_topk_kernel<TC_BF16, true, 1>, gp, mp)
               : a.mode == TC_FP8 ? run(tc_topk_kernel<TC_FP8, true, 1>, gp, mp)
                                  : run(tc_topk_kernel<TC_SIGN, true, 1>, gp, mp));
        tc_bound_kernel<<<(unsigned)ceil_div(a.nq, 8), 256, 0, st>>>(s.gmin, (TC_NEPI / 4) * p.pilot_chunks, a.nq,
                                                                    a.bound_rank ? a.bound_rank : a.S, a.slack,
                                                                    s.qbound);
    } else {
        GN_CUDA_TRY(cudaMemsetAsync(s.qbound, 0xff, (size_t)a.nq * 4, st));
    }
    s.nchunks = p.nchunks;
    s.ntiles = ceil_div(a.n, TC_N);
    s.n = a.n;
    s.bnorm = a.bnorm;
    s.bscale = a.bscale;
    if (g.qt == 2)
        return a.mode == TC_BF16  ? run(tc_topk_kernel<TC_BF16, false, 2>, g, mb)
               : a.mode == TC_FP8 ? run(tc_topk_kernel<TC_FP8, false, 2>, g, mb)
                                  : run(tc_topk_kernel<TC_SIGN, false, 2>, g, mb);
    return a.mode == TC_BF16  ? run(tc_topk_kernel<TC_BF16, false, 1>, g, mb)
           : a.mode == TC_FP8 ? run(tc_topk_kernel<TC_FP8, false, 1>, g, mb)
                              : run(tc_topk_kernel<TC_SIGN, false, 1>, g, mb);
}

// ── conversion and norms ──────────────────────────────────────────────────
__global__ void f32_to_bf16_rows_kernel(const float *__restrict__ X, int64_t n, int d, int ldx,
                                        __nv_bfloat16 *__restrict__ out, int K) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * K) return;
    const int64_t i = t / K;
    const int j = (int)(t % K);
    out[t] = __float2bfloat16_rn(j < d ? X[i * ldx + j] : 0.f);
}

void to_bf16_rows(const float *X, int64_t n, int d, int ldx, void *out, int K, cudaStream_t st) {
    if (n > 0)
        f32_to_bf16_rows_kernel<<<(unsigned)ceil_div(n * K, 256), 256, 0, st>>>(
            X, n, d, ldx, reinterpret_cast<__nv_bfloat16 *>(out), K);
}

// FP8 E4M3 rows with one FP32 scale each: warp per row; scale = max|x| / 448
// (the largest E4M3 magnitude; 1 for an all-zero row), element = x / scale
// rounded to nearest E4M3 with saturation, zero beyond d up to K.
__global__ void f32_to_e4m3_rows_kernel(const float *__restrict__ X, int64_t n, int d, int ldx,
                                        uint8_t *__restrict__ out, float *__restrict__ scale, int K) {
    const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    const float *x = X + r * ldx;
    float m = 0.f;
    for (int j = lane; j < d; j += 32) m = fmaxf(m, fabsf(x[j]));
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float sc = m > 0.f ? m / 448.f : 1.f;
    const float inv = m > 0.f ? 448.f / m : 1.f;
    if (lane == 0) scale[r] = sc;
    uint8_t *o = out + r * K;
    for (int j = lane; j < K; j += 32)
        o[j] = j < d ? (uint8_t)__nv_cvt_float_to_fp8(x[j] * inv, __NV_SATFINITE, __NV_E4M3) : (uint8_t)0;
}

void to_e4m3_rows(const float *X, int64_t n, int d, int ldx, void *out, float *scale, int K, cudaStream_t st) {
    if (n > 0)
        f32_to_e4m3_rows_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, st>>>(X, n, d, ldx,
                                                                          reinterpret_cast<uint8_t *>(out), scale, K);
}

// ── exact re-rank ─────────────────────────────────────────────────────────
// The k nearest (k <= 32) of m candidate keys' rows to query q, by one warp, in
// the reference's FP32 order (bit-identical to the exact flat scan).  Two lanes
// per row, each with four of the reference's eight accumulators, so a warp's
// loads take whole 32-byte sectors of 16 rows.
__device__ __forceinline__ void l2_rank(const uint64_t *keys, int m, const float *__restrict__ q,
                                        const float *__restrict__ X, int d, int dp, int k,
                                        int64_t *__restrict__ out_idx, float *__restrict__ out_dist) {
    const int lane = threadIdx.x & 31;
    const float4 *q4 = reinterpret_cast<const float4 *>(q);
    const int half = lane & 1;
    const int nb = d >> 3, rem = d & 7;
    WarpTopK<1> F;
    F.init();
    uint64_t fthr = KEY_EMPTY;
    for (int c0 = 0; c0 < m; c0 += 16) {
        const int c = c0 + (lane >> 1);
        const bool in = c < m;
        const uint32_t row = key_idx(keys[in ? c : 0]);
        const float4 *x4 = reinterpret_cast<const float4 *>(X + (int64_t)row * dp);
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll 8
        for (int b = 0; b < nb; ++b) {
            const float4 x = x4[2 * b + half], y = q4[2 * b + half];
            const float t0 = __fsub_rn(y.x, x.x), t1 = __fsub_rn(y.y, x.y);
            const float t2 = __fsub_rn(y.z, x.z), t3 = __fsub_rn(y.w, x.w);
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
            const float4 x = x4[2 * nb + w], y = q4[2 * nb + w];
            const float t0 = __fsub_rn(y.x, x.x), t1 = __fsub_rn(y.y, x.y);
            const float t2 = __fsub_rn(y.z, x.z), t3 = __fsub_rn(y.w, x.w);
            s0 = __fmaf_rn(t0, t0, s0);
            s1 = __fmaf_rn(t1, t1, s1);
            s2 = __fmaf_rn(t2, t2, s2);
            s3 = __fmaf_rn(t3, t3, s3);
        }
        const float dd = __fsqrt_rn(__fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2, s3)));
        F.offer(in && half == 0 ? make_key(__float_as_uint(dd), row) : KEY_EMPTY, fthr, k);
    }
    if (lane < k) {
        const uint64_t key = F.v[0];
        const bool e = key == KEY_EMPTY;
        out_idx[lane] = e ? -1 : (int64_t)key_idx(key);
        out_dist[lane] = e ? 0.f : __uint_as_float(key_dist(key));
    }
}

// One warp per query: the S best candidates by score, then the k nearest of them.
constexpr int RR_WARPS = 4;
__global__ void __launch_bounds__(RR_WARPS * 32)
    tc_rerank_kernel(const uint64_t *__restrict__ part, const int *__restrict__ qcount, int64_t slot_keys, int S,
                     const float *__restrict__ Q, const float *__restrict__ X, int d, int dp, int64_t nq, int k,
                     int64_t *__restrict__ out_idx, float *__restrict__ out_dist) {
    __shared__ uint64_t s_sel[RR_WARPS][64];
    const int warp = threadIdx.x >> 5;
    const int64_t q = (int64_t)blockIdx.x * RR_WARPS + warp;
    if (q >= nq) return;
    const int m = warp_best(part + q * slot_keys, qcount[q], S, s_sel[warp]);
    l2_rank(s_sel[warp], m, Q + q * dp, X, d, dp, k, out_idx + q * k, out_dist + q * k);
}

// ── exact Hamming k-NN of large batches ───────────────────────────────────
// Packed rows -> E4M3 +1 (bit set) / -1 (clear), 0 past the row's bits: a thread
// per 16 bits.
__global__ void bits_to_signs_kernel(const uint16_t *__restrict__ X, int64_t n, int pitch16, int nbits,
                                     uint4 *__restrict__ out, int K) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int per = K / 16;
    if (t >= n * per) return;
    const int64_t r = t / per;
    const int h = (int)(t % per);
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (h * 16 < nbits) {
        const uint32_t bits = X[r * pitch16 + h];
        const int valid = min(16, nbits - h * 16);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (i < valid) w[i >> 2] |= ((bits >> i) & 1u ? 0x38u : 0xB8u) << (8 * (i & 3));
    }
    out[t] = make_uint4(w[0], w[1], w[2], w[3]);
}

// The k nearest of each query's candidates ((h, row) keys), by one warp.
__global__ void __launch_bounds__(RR_WARPS * 32)
    ham_finish_kernel(const uint64_t *__restrict__ part, const int *__restrict__ qcount, int64_t slot_keys,
                      int64_t nq, int k, int64_t *__restrict__ out_idx, int64_t *__restrict__ out_dist) {
    __shared__ uint64_t s_sel[RR_WARPS][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t q = (int64_t)blockIdx.x * RR_WARPS + warp;
    if (q >= nq) return;
    const int m = warp_best(part + q * slot_keys, qcount[q], k, s_sel[warp]);
    uint64_t v[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) v[r] = r * 32 + lane < m ? s_sel[warp][r * 32 + lane] : KEY_EMPTY;
    warp_sort<2>(v);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int p = r * 32 + lane;
        if (p >= k) continue;
        const bool e = v[r] == KEY_EMPTY;
        out_idx[q * k + p] = e ? -1 : (int64_t)key_idx(v[r]);
        out_dist[q * k + p] = e ? 0 : (int64_t)key_dist(v[r]);
    }
}

// Expanded operands and scratch of a Hamming index, made by its first large search.
struct HamTc {
    DBuf x8, q8, part, qcount;
    TcScratch scr;
    bool built = false, refused = false;
};

// Where the tensor cores answer a Hamming search.  Both paths give the same
// results; the sums of +-1 products are whole numbers of at most 4,096, exact in
// any accumulator.  Measured per 1e10 pairs of 512 bits: 36.5 ms on the POPC
// scan, 4.1 ms here; the expanded rows cost 8 bytes per packed byte, the
// batch is padded to whole tiles of 128 queries and the pilot, the selection
// and the launches take some 60 to 100 us.  So batches below 128 queries stay on
// the POPC scan, and those of less than half a millisecond there (2 G words; or,
// where the expanded rows are small enough for the first search to make them in
// passing, half of that or 62 M pairs, which cost the POPC scan's selection as much:
// 31,361 x 160 bits, 3,585 queries, k 3: 410 us a search there, 189 here).
bool ham_tc_wanted(const gn_index *ix, int64_t nq, int64_t k) {
    const int64_t words = ceil_div(ix->dim, 4);
    const bool small = ix->n * round_up(ix->dim * 8, TC_BK8) <= (int64_t)128 << 20;
    const int64_t weight = small ? std::max<int64_t>(2 * words, 32) : words;
    return k <= 64 && ix->dim <= 512 && ix->n >= TC_EXACT_MIN && nq >= 128 && nq * ix->n >= 2000000000ll / weight;
}

// Returns GN_ERR_UNSUPPORTED where the expanded rows do not fit (the caller
// then uses the POPC scan).
int ham_tc_search(gn_index *ix, const void *d_q, int64_t nq, int k, int64_t *d_idx, int64_t *d_dist, int *err,
                  cudaStream_t st) {
    if (!ix->ext) {
        ix->ext = new HamTc();
        ix->ext_free = [](void *p) { delete reinterpret_cast<HamTc *>(p); };
    }
    HamTc &H = *reinterpret_cast<HamTc *>(ix->ext);
    if (H.refused) return GN_ERR_UNSUPPORTED;
    const int nbits = (int)ix->dim * 8, pitch16 = ix->stride4 * 8;
    const int K = (int)round_up(nbits, TC_BK8);
    auto expand = [&](const void *x, int64_t n, DBuf &out) {
        bits_to_signs_kernel<<<(unsigned)ceil_div(n * (K / 16), 256), 256, 0, st>>>(
            reinterpret_cast<const uint16_t *>(x), n, pitch16, nbits, out.as<uint4>(), K);
    };
    if (!H.built) {
        // at most a quarter of the free memory for the expanded rows
        size_t free_b = 0, total_b = 0;
        const size_t want = (size_t)std::max<int64_t>(ix->n, TC_N) * K;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || want > free_b / 4 || H.x8.ensure(want) != GN_OK) {
            cudaGetLastError();
            H.refused = true;  // until the next set()
            return GN_ERR_UNSUPPORTED;
        }
        expand(ix->data.p, ix->n, H.x8);
        H.built = true;
    }
    for (int64_t b0 = 0; b0 < nq; b0 += TC_QBLOCK) {
        const int64_t bq = std::min<int64_t>(TC_QBLOCK, nq - b0);
        // (lists of at least 16: with fewer, rows tied at the last distance would have them
        // sorted; 15,000 x 8 bits, 9,000 queries, k 1: 426 us, 197 so)
        const int S = std::max(k, 16);
        const TcPlan plan = tc_plan(TC_SIGN, K, bq, ix->n, S);
        if (H.q8.ensure((size_t)std::max<int64_t>(bq, TC_M) * K) != GN_OK ||
            H.part.ensure((size_t)bq * plan.slot_keys * 8) != GN_OK || H.qcount.ensure((size_t)bq * 4) != GN_OK)
            return GN_ERR_UNSUPPORTED;
        expand(static_cast<const uint8_t *>(d_q) + (size_t)b0 * ix->stride4 * 16, bq, H.q8);
        TcLaunch a;
        a.mode = TC_SIGN;
        a.A = H.q8.p;
        a.nq = bq;
        a.a_rows = std::max<int64_t>(bq, TC_M);
        a.B = H.x8.p;
        a.n = ix->n;
        a.b_rows = std::max<int64_t>(ix->n, TC_N);
        a.K = K;
        a.nbits = nbits;
        a.part = H.part.as<uint64_t>();
        a.qcount = H.qcount.as<int>();
        a.err = err;
        a.S = S;
        a.bound_rank = k;
        timing_begin(st, "tc_topk_kernel");
        const int rc = tc_topk_launch(a, plan, H.scr, st);
        timing_end(st);
        if (rc != GN_OK) return rc == GN_ERR_OOM ? (int)GN_ERR_UNSUPPORTED : rc;
        ham_finish_kernel<<<(unsigned)ceil_div(bq, RR_WARPS), RR_WARPS * 32, 0, st>>>(
            H.part.as<uint64_t>(), H.qcount.as<int>(), plan.slot_keys, bq, k, d_idx + b0 * k, d_dist + b0 * k);
    }
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

// ── exact L2 k-NN of large batches ────────────────────────────────────────
// The exact scan's answer (indices, and distances bit for bit) through the
// tensor cores.  Each FP32 value is split into two BF16 parts, v = hi + lo + r with
// |lo| <= L |v| and |r| <= L^2 |v|, L = 2^-8 (BF16 keeps eight significant bits), and
// rows are laid out as [hi | lo | hi], the query as [hi | hi | lo], so that one GEMM
// sums hi hi + hi lo + lo hi.  Left out are lo lo, r times a row's value and a query's
// hi + lo times r: (3 + L^2) L^2 |q||x| at most.  The score a = |x|^2 - 2 acc then differs
// from D - |q|^2 (D the squared distance in exact arithmetic) by at most
//     E = cross |q| max|x| + norm max|x|^2:
// cross = 2 (SPLIT_LEFT + u), u |q||x| for the FP32 sums of K terms in the tensor
// core, for which u = 2^-14 per 512 terms is allowed, a thousand roundings of 2^-24
// each; norm: the row norms' own FP32 sums.
//
// The pilot gives B, a score that k rows reach.  Their D is at most B + |q|^2 +
// E, and the FP32 distance of any row lies within a relative g = (d / 8 + 16) 2^-23
// of its D (the eight-accumulator sums, the differences' roundings, the root, and
// distances that tie after it), so a row among the k nearest has D <= (B + |q|^2 +
// E)(1 + rel), rel = 4 g, hence a score of at most B + 2 E + rel (B + |q|^2 + E).
// Every row up to that bound is kept, its distance computed in the reference's
// order, and the k nearest returned.  If some buffer could not hold its rows (many
// ties, or values so large against their differences that E spans most rows),
// a flag is set and the FP32 scan, launched behind it, answers instead (it ends
// at once when the flag is clear).  One such search says little (a query that is not
// a number is enough), several in a row that the rows are not for this path: see
// l2_tc_given_up.
constexpr float SPLIT_LO = 0x1p-8f;                              // L
constexpr float SPLIT_LEFT = 3.01f * SPLIT_LO * SPLIT_LO;        // the products left out, of |q||x|
__global__ void split_rows_kernel(const float *__restrict__ X, int64_t n, int d, int ldx, bool query,
                                  __nv_bfloat16 *__restrict__ out, int K) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * K) return;
    const int64_t i = t / K;
    const int j = (int)(t % K), part = j / d;  // part 3: padding
    __nv_bfloat16 v = __float2bfloat16_rn(0.f);
    if (part < 3) {
        const float x = X[i * ldx + (j - part * d)];
        const __nv_bfloat16 hi = __float2bfloat16_rn(x);
        const bool low = part == (query ? 2 : 1);
        v = low ? __float2bfloat16_rn(__fsub_rn(x, __bfloat162float(hi))) : hi;
    }
    out[t] = v;
}

__global__ void max_value_kernel(const float *__restrict__ x, int64_t n, uint32_t *__restrict__ out) {
    float m = 0.f;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = fmaxf(m, x[i]);
    const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if ((threadIdx.x & 31) == 0) atomicMax(out, w);
}

// One warp per query: the distances of all its candidates, the k nearest.
__global__ void __launch_bounds__(RR_WARPS * 32)
    l2_finish_kernel(const uint64_t *__restrict__ part, const int *__restrict__ qcount, int64_t slot_keys,
                     const float *__restrict__ Q, const float *__restrict__ X, int d, int dp, int64_t nq, int k,
                     int64_t *__restrict__ out_idx, float *__restrict__ out_dist, int *flag) {
    const int64_t q = (int64_t)blockIdx.x * RR_WARPS + (threadIdx.x >> 5);
    if (q >= nq) return;
    // fewer candidates than results: rows whose scores are not numbers
    if ((threadIdx.x & 31) == 0 && qcount[q] < k) *flag = 1;
    l2_rank(part + q * slot_keys, qcount[q], Q + q * dp, X, d, dp, k, out_idx + q * k, out_dist + q * k);
}

// Split operands and scratch of an L2 index, made by its large searches.
struct L2Tc {
    HBuf hflag;  // the flag of the last search done, -1 once it is counted (freed after the device buffers)
    DBuf x16, xnorm, pnorm, xmax2, q16, qnorm, part, qcount, flag;
    TcScratch scr;
    bool built = false, refused = false;
    int overflows = 0, passed_by = 0;  // searches in a row that set the flag, and searches since then
    double seen = 0.0;                 // what searches had to gain from split rows, in elements of the FP32 scan
};
static L2Tc &l2_tc_state(gn_index *ix) {
    if (!ix->ext) {
        ix->ext = new L2Tc();
        ix->ext_free = [](void *p) { delete reinterpret_cast<L2Tc *>(p); };
    }
    return *reinterpret_cast<L2Tc *>(ix->ext);
}

// The FP32 scan alone answers where it had to answer L2TC_OVERFLOWS searches in a row,
// but for every L2TC_RETRY-th search: a batch of odd queries is forgotten again, and
// rows that never fit cost a 32nd of the tensor-core scan's time at most.
constexpr int L2TC_OVERFLOWS = 4, L2TC_RETRY = 32;
static bool l2_tc_given_up(L2Tc &H) {
    if (!H.hflag.p) return false;
    volatile int *word = reinterpret_cast<volatile int *>(H.hflag.p);
    const int flag = *word;  // (a copy that lands in between is not counted)
    if (flag >= 0) {
        H.overflows = flag ? H.overflows + 1 : 0;
        *word = -1;
    }
    if (H.overflows < L2TC_OVERFLOWS) return false;
    return ++H.passed_by % L2TC_RETRY != 0;
}

// Where the tensor cores answer an exact L2 search: measured for 100k x 32, 1,000
// queries, k 5: 416 us on the FP32 scan, 148 us the whole call here, of which 60 us do
// not depend on the size; the FP32 scan takes about 0.13 ns per element, so
// batches of less than 1.5 G elements stay there, and small ones, which fill
// a part of a 128-query tile.
// The split rows are made once the searches of these rows have had about as much to
// gain from them as they cost.  A search gains the FP32 scan's time less some 0.8 G
// elements' worth; making the rows takes about 27 elements' time a byte (0.4 TB/s, most of
// it the allocation) and, with the scratch of an index's first search, 1.6 G elements' (0.8 G
// later).  First searches after set(), in us, always here / on the FP32 scan / with
// this rule: 20,000 x 64 rows, 1,200 queries 577 / 413 / 413; 200,000 x 128, 64 queries
// 741 / 318 / 318 (later searches 215 and 253); 100,000 x 32, 1,000 queries 552 / 612 / 552.
bool l2_tc_wanted(gn_index *ix, int64_t nq, int64_t k) {
    if (k > 32 || ix->n < TC_EXACT_MIN || nq < 64 || ix->dim > 2048) return false;
    const double work = (double)nq * (double)ix->n * (double)ix->dim;
    if (work < 1.5e9) return false;
    L2Tc &H = l2_tc_state(ix);
    if (H.refused) return false;
    if (!H.built) {
        const double bytes = (double)ix->n * (double)round_up(3 * ix->dim, TC_BK) * 2.0;
        H.seen += work - 0.8e9;
        return H.seen >= (H.part.p ? 0.8e9 : 1.6e9) + 27.0 * bytes;
    }
    return !l2_tc_given_up(H);
}

// On success *flag is the device word that tells whether the results stand (0) or
// the caller's FP32 scan has to answer.  GN_ERR_UNSUPPORTED: nothing was
// launched that the caller needs to know of.
int l2_tc_search(gn_index *ix, const float *d_q, int64_t nq, int k, int64_t *d_idx, float *d_dist, int *err,
                 const int **flag, cudaStream_t st) {
    L2Tc &H = l2_tc_state(ix);
    const int d = (int)ix->dim, dp = ix->stride4 * 4;
    const int K = (int)round_up(3 * d, TC_BK);
    const float *x32 = ix->data.as<float>();
    auto split = [&](const float *x, int64_t n, bool query, DBuf &out) {
        split_rows_kernel<<<(unsigned)ceil_div(n * K, 256), 256, 0, st>>>(x, n, d, dp, query,
                                                                         out.as<__nv_bfloat16>(), K);
    };
    if (!H.built) {
        // at most a quarter of the free memory for the split rows
        size_t free_b = 0, total_b = 0;
        const size_t want = (size_t)ix->n * K * 2, np = (size_t)round_up(ix->n, TC_N);
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || want > free_b / 4 || H.x16.ensure(want) != GN_OK ||
            H.xnorm.ensure(np * 4) != GN_OK || H.pnorm.ensure(tc_pilot_count(ix->n) * 4) != GN_OK ||
            H.xmax2.ensure(4) != GN_OK || H.flag.ensure(4) != GN_OK || H.hflag.ensure(4) != GN_OK) {
            cudaGetLastError();
            H.refused = true;  // until the next set()
            return GN_ERR_UNSUPPORTED;
        }
        *reinterpret_cast<volatile int *>(H.hflag.p) = -1;
        split(x32, ix->n, false, H.x16);
        GN_CUDA_TRY(cudaMemsetAsync(H.xnorm.as<float>() + ix->n, 0xff, (np - (size_t)ix->n) * 4, st));
        row_norms(x32, ix->n, dp, H.xnorm.as<float>(), st);
        GN_TRY(tc_pilot_values(H.xnorm.as<float>(), ix->n, H.pnorm, st));
        GN_CUDA_TRY(cudaMemsetAsync(H.xmax2.p, 0, 4, st));
        max_value_kernel<<<256, 256, 0, st>>>(H.xnorm.as<float>(), ix->n, H.xmax2.as<uint32_t>());
        H.built = true;
    }
    GN_CUDA_TRY(cudaMemsetAsync(H.flag.p, 0, 4, st));
    for (int64_t b0 = 0; b0 < nq; b0 += L2TC_QBLOCK) {
        const int64_t bq = std::min<int64_t>(L2TC_QBLOCK, nq - b0);
        const float *bx = d_q + b0 * dp;
        const TcPlan plan = tc_plan(TC_BF16, K, bq, ix->n, TC_CAP - 32);
        const int64_t a_rows = std::max<int64_t>(bq, TC_M);
        if (H.q16.ensure((size_t)a_rows * K * 2) != GN_OK || H.qnorm.ensure((size_t)bq * 4) != GN_OK ||
            H.part.ensure((size_t)bq * plan.slot_keys * 8) != GN_OK || H.qcount.ensure((size_t)bq * 4) != GN_OK)
            return GN_ERR_UNSUPPORTED;
        split(bx, bq, true, H.q16);
        row_norms(bx, bq, dp, H.qnorm.as<float>(), st);
        TcLaunch a;
        a.mode = TC_BF16;
        a.A = H.q16.p;
        a.nq = bq;
        a.a_rows = a_rows;
        a.B = H.x16.p;
        a.n = ix->n;
        a.b_rows = ix->n;
        a.K = K;
        a.bnorm = H.xnorm.as<float>();
        a.pnorm = H.pnorm.as<float>();
        a.part = H.part.as<uint64_t>();
        a.qcount = H.qcount.as<int>();
        a.err = err;
        a.S = TC_CAP - 32;
        a.bound_rank = k;
        a.overflow = H.flag.as<int>();
        const float g = (float)(d / 8 + 16) * 0x1p-23f;
        a.slack.q2 = H.qnorm.as<float>();
        a.slack.xmax2 = H.xmax2.as<uint32_t>();
        a.slack.overflow = H.flag.as<int>();
        a.slack.cross = 2.f * (SPLIT_LEFT + 0x1p-14f * (float)ceil_div(K, 512));
        a.slack.norm = (float)(d / 32 + 16) * 0x1p-23f;
        a.slack.rel = 4.f * g;
        timing_begin(st, "tc_topk_kernel");
        const int rc = tc_topk_launch(a, plan, H.scr, st);
        timing_end(st);
        if (rc != GN_OK) return rc == GN_ERR_OOM ? (int)GN_ERR_UNSUPPORTED : rc;
        l2_finish_kernel<<<(unsigned)ceil_div(bq, RR_WARPS), RR_WARPS * 32, 0, st>>>(
            H.part.as<uint64_t>(), H.qcount.as<int>(), plan.slot_keys, bx, x32, d, dp, bq, k, d_idx + b0 * k,
            d_dist + b0 * k, H.flag.as<int>());
    }
    GN_CUDA_TRY(cudaMemcpyAsync(H.hflag.p, H.flag.p, 4, cudaMemcpyDeviceToHost, st));
    *flag = H.flag.as<int>();
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

void flat_tc_reset(gn_index *ix) {
    if (!ix->ext) return;
    if (ix->metric == M_HAMMING) {
        HamTc &H = *reinterpret_cast<HamTc *>(ix->ext);
        H.built = H.refused = false;
        H.x8.release();
    } else {
        L2Tc &H = *reinterpret_cast<L2Tc *>(ix->ext);
        H.built = H.refused = false;
        H.overflows = H.passed_by = 0;
        H.seen = 0.0;
        H.x16.release();  // (waits for the searches queued, and with them for their flags' copies)
        if (H.hflag.p) *reinterpret_cast<volatile int *>(H.hflag.p) = -1;
    }
}

// ── flat tensor-core index (exact L2 via shortlist + re-rank) ─────────────
struct TcFlatState {
    int d = 0, dp = 0, K = 0;
    int S = 40;
    int fp8 = 0;  // 0: BF16 operands; 1: FP8 E4M3 with per-row scales
    int64_t n = 0;
    DBuf x32, x16, xnorm, xscale;  // fp32 rows (dp), low-precision rows (K), |x|^2, FP8 row scales
    DBuf pnorm, pscale;            // norms and scales of the pilot's rows
    DBuf q32, q16, qscale, part, qcount, err, out_idx, out_dist;
    TcScratch scr;
};

// The database's low-precision copy in the index's precision, from its FP32
// rows; it holds at least one full 256-row TMA box.
static int tcflat_lowp(TcFlatState &S, cudaStream_t st) {
    S.K = (int)round_up(S.d, S.fp8 ? TC_BK8 : TC_BK);
    const size_t bytes = (size_t)std::max<int64_t>(S.n, TC_N) * S.K * (S.fp8 ? 1 : 2);
    GN_TRY(S.x16.ensure(bytes));
    GN_CUDA_TRY(cudaMemsetAsync(S.x16.p, 0, bytes, st));
    if (S.fp8) {
        GN_TRY(S.xscale.ensure((size_t)round_up(S.n, TC_N) * 4));  // whole tiles are read
        to_e4m3_rows(S.x32.as<float>(), S.n, S.d, S.dp, S.x16.p, S.xscale.as<float>(), S.K, st);
        GN_TRY(tc_pilot_values(S.xscale.as<float>(), S.n, S.pscale, st));
    } else {
        S.xscale.release();
        to_bf16_rows(S.x32.as<float>(), S.n, S.d, S.dp, S.x16.p, S.K, st);
    }
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

}  // namespace gn

using namespace gn;

static TcFlatState *tcs(gn_index *ix) { return reinterpret_cast<TcFlatState *>(ix->ext); }

extern "C" {

int gn_tcflat_create(int32_t shortlist, gn_index **out) {
    if (!out) return fail(GN_ERR_INVALID, "out is NULL");
    if (shortlist != 16 && shortlist != 32 && shortlist != 40 && shortlist != 48 && shortlist != 56 &&
        shortlist != 64)
        return fail(GN_ERR_INVALID, "shortlist must be 16, 32, 40, 48, 56 or 64");
    gn_index *ix = new gn_index();
    ix->kind = K_TCFLAT;
    ix->metric = GN_METRIC_L2;
    TcFlatState *S = new TcFlatState();
    S->S = shortlist;
    ix->ext = S;
    ix->ext_free = [](void *p) { delete reinterpret_cast<TcFlatState *>(p); };
    *out = ix;
    return GN_OK;
}

int gn_tcflat_set(gn_index *ix, const float *data, int64_t n, int64_t d) {
    if (!ix || ix->kind != K_TCFLAT) return fail(GN_ERR_INVALID, "not a tensor-core flat index");
    if (n <= 0 || d <= 0 || !data) return fail(GN_ERR_INVALID, "data must be a non-empty (N, D) array");
    if (n >= 0x7fffffffLL) return fail(GN_ERR_UNSUPPORTED, "at most 2^31-2 rows");
    std::lock_guard<std::mutex> lk(ix->mu);
    GN_TRY(make_stream(ix));
    TcFlatState &S = *tcs(ix);
    cudaStream_t st = ix->stream;
    S.n = n;
    S.d = (int)d;
    S.dp = (int)round_up(d, 4);
    GN_TRY(upload_rows(S.x32, data, n, d * 4, S.dp / 4, st));
    // |x|^2 in FP32, up to whole tiles: NaN past the last row
    const size_t np = (size_t)round_up(n, TC_N);
    GN_TRY(S.xnorm.ensure(np * 4));
    GN_CUDA_TRY(cudaMemsetAsync(S.xnorm.as<float>() + n, 0xff, (np - (size_t)n) * 4, st));
    row_norms(S.x32.as<float>(), n, S.dp, S.xnorm.as<float>(), st);
    GN_TRY(tc_pilot_values(S.xnorm.as<float>(), n, S.pnorm, st));
    GN_TRY(tcflat_lowp(S, st));
    GN_TRY(S.err.ensure(4));
    GN_CUDA_TRY(cudaMemsetAsync(S.err.p, 0, 4, st));
    GN_CUDA_TRY(cudaStreamSynchronize(st));
    GN_CUDA_TRY(cudaGetLastError());
    ix->n = n;
    ix->dim = d;
    return GN_OK;
}

// Argument checks shared by the device- and host-buffer searches.
static int tcflat_check(gn_index *ix, int64_t k) {
    if (!ix || ix->kind != K_TCFLAT) return fail(GN_ERR_INVALID, "not a tensor-core flat index");
    TcFlatState &S = *tcs(ix);
    if (S.n == 0) return fail(GN_ERR_EMPTY, "index is empty");
    if (k <= 0 || k > 32 || k > S.S) return fail(GN_ERR_INVALID, "k must be in [1, min(32, shortlist)]");
    return GN_OK;
}

// The search on device buffers, with the index's lock held by the caller.
static int tcflat_search_locked(gn_index *ix, const float *d_queries, int64_t nq, int64_t k, int64_t *d_idx,
                                float *d_dist, cudaStream_t st) {
    TcFlatState &S = *tcs(ix);
    for (int64_t b0 = 0; b0 < nq; b0 += TC_QBLOCK) {
        const int64_t bq = std::min<int64_t>(TC_QBLOCK, nq - b0);
        const float *bx = d_queries + b0 * S.dp;
        const TcPlan plan = tc_plan(S.fp8 ? TC_FP8 : TC_BF16, S.K, bq, S.n, S.S);
        const int64_t a_rows = std::max<int64_t>(bq, TC_M);  // >= one 128-row TMA box
        GN_TRY(S.q16.ensure((size_t)a_rows * S.K * (S.fp8 ? 1 : 2)));
        GN_TRY(S.part.ensure((size_t)bq * plan.slot_keys * 8));
        GN_TRY(S.qcount.ensure((size_t)bq * 4));
        if (S.fp8) {
            GN_TRY(S.qscale.ensure((size_t)bq * 4));
            to_e4m3_rows(bx, bq, S.d, S.dp, S.q16.p, S.qscale.as<float>(), S.K, st);
        } else {
            to_bf16_rows(bx, bq, S.d, S.dp, S.q16.p, S.K, st);
        }
        TcLaunch a;
        a.mode = S.fp8 ? TC_FP8 : TC_BF16;
        a.A = S.q16.p;
        a.nq = bq;
        a.a_rows = a_rows;
        a.B = S.x16.p;
        a.n = S.n;
        a.b_rows = std::max<int64_t>(S.n, TC_N);
        a.K = S.K;
        a.bnorm = S.xnorm.as<float>();
        a.pnorm = S.pnorm.as<float>();
        a.part = S.part.as<uint64_t>();
        a.qcount = S.qcount.as<int>();
        a.err = S.err.as<int>();
        a.S = S.S;
        a.ascale = S.fp8 ? S.qscale.as<float>() : nullptr;
        a.bscale = S.fp8 ? S.xscale.as<float>() : nullptr;
        a.pscale = S.fp8 ? S.pscale.as<float>() : nullptr;
        timing_begin(st, "tc_topk_kernel");
        GN_TRY(tc_topk_launch(a, plan, S.scr, st));
        timing_end(st);
        tc_rerank_kernel<<<(unsigned)ceil_div(bq, RR_WARPS), RR_WARPS * 32, 0, st>>>(
            S.part.as<uint64_t>(), S.qcount.as<int>(), plan.slot_keys, S.S, bx, S.x32.as<float>(), S.d, S.dp, bq,
            (int)k, d_idx + b0 * k, d_dist + b0 * k);
    }
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

int gn_tcflat_search_knn_device(gn_index *ix, const float *d_queries, int64_t nq, int64_t k, int64_t *d_idx,
                                float *d_dist, void *stream) {
    GN_TRY(tcflat_check(ix, k));
    if (nq <= 0) return GN_OK;
    std::lock_guard<std::mutex> lk(ix->mu);
    return tcflat_search_locked(ix, d_queries, nq, k, d_idx, d_dist, (cudaStream_t)stream);
}

int gn_tcflat_search_knn(gn_index *ix, const float *queries, int64_t nq, int64_t k, int64_t *out_idx,
                         float *out_dist) {
    GN_TRY(tcflat_check(ix, k));
    if (nq < 0 || (nq > 0 && (!queries || !out_idx || !out_dist))) return fail(GN_ERR_INVALID, "bad arguments");
    if (nq == 0) return GN_OK;
    TcFlatState &S = *tcs(ix);
    cudaStream_t st = ix->stream;
    // the lock covers the whole call: the query, result and staging buffers are the index's
    std::lock_guard<std::mutex> lk(ix->mu);
    begin_blocking(ix);
    GN_TRY(upload_queries(ix, S.q32, queries, nq, S.d * 4, S.dp / 4, st));
    void *d_idx = nullptr, *d_dist = nullptr;
    GN_TRY(place_result(ix, S.out_idx, out_idx, (size_t)nq * k * 8, &d_idx));
    GN_TRY(place_result(ix, S.out_dist, out_dist, (size_t)nq * k * 4, &d_dist));
    GN_TRY(tcflat_search_locked(ix, S.q32.as<float>(), nq, k, static_cast<int64_t *>(d_idx),
                                static_cast<float *>(d_dist), st));
    GN_TRY(download_result(ix, out_idx, d_idx, (size_t)nq * k * 8, st));
    GN_TRY(download_result(ix, out_dist, d_dist, (size_t)nq * k * 4, st));
    return finish_blocking(ix, S.err.as<int>(), st, "tensor-core scan: a pipeline wait timed out");
}

int gn_tcflat_set_precision(gn_index *ix, int32_t precision) {
    if (!ix || ix->kind != K_TCFLAT) return fail(GN_ERR_INVALID, "not a tensor-core flat index");
    if (precision != 0 && precision != 1) return fail(GN_ERR_INVALID, "precision must be 0 (BF16) or 1 (FP8 E4M3)");
    std::lock_guard<std::mutex> lk(ix->mu);
    TcFlatState &S = *tcs(ix);
    if (precision == 1 && S.S > 56)
        return fail(GN_ERR_UNSUPPORTED, "FP8 shortlist: S must be 16, 32, 40, 48 or 56");
    if (S.fp8 == precision) return GN_OK;
    S.fp8 = precision;
    if (S.n > 0) {
        GN_TRY(tcflat_lowp(S, ix->stream));
        GN_CUDA_TRY(cudaStreamSynchronize(ix->stream));
    }
    return GN_OK;
}

int gn_tc_error(gn_index *ix, int32_t *err_out) {
    if (!ix || ix->kind != K_TCFLAT) return fail(GN_ERR_INVALID, "not a tensor-core flat index");
    int herr = 0;
    GN_CUDA_TRY(cudaMemcpy(&herr, tcs(ix)->err.p, 4, cudaMemcpyDeviceToHost));
    if (err_out) *err_out = herr;
    return GN_OK;
}

}  // extern "C"
