// gemm_topk.cuh — FP32 CUDA-core tile GEMM for fused selection epilogues.
//
// One CTA of 256 threads multiplies a tile of BM=64 "A" rows (queries or
// points, gathered through an index list) with tiles of 128 H "B" rows
// (centroids or database rows, contiguous) over K = dp (a multiple of 16,
// zero padded).  Thread t owns A rows 8*(t/32) .. +8 and, in each half of 128 B
// rows, rows 4*(t%32) .. +4, so warp w owns eight whole A rows across the full B
// tile: a fused epilogue can select for the warp's rows without staging the
// scores through shared memory.
//
// Each product is one fused multiply-add in ascending k, two per instruction
// (f32x2.cuh).  The A tile is stored with every value twice, so that a pair
// operand is one shared load; with H = 2 a step of k takes 12 shared-memory
// wavefronts per warp for 64 cycles of the FP32 pipe (H = 1: 8 for 32, the
// shared-memory pipe's whole rate).  The next slice of K is held in registers
// while the current one is multiplied.  100k x 64 against 256 centroids: 102 us
// with scalar products and slices stored as they arrived, 92 us (the pairs keep
// the FP32 pipe half busy; four slices per tile leave the first load exposed).
#pragma once

#include "common.cuh"
#include "f32x2.cuh"

namespace gn {

constexpr int GT_BM = 64, GT_BN = 128, GT_BK = 16, GT_THREADS = 256;

template <int H>
struct GemmTileSmem {
    float2 As[2][GT_BK][GT_BM + 2];
    float Bs[2][GT_BK][GT_BN * H + 4];
};

// Orderable transform of a float (total order, negatives below positives).
__device__ __forceinline__ uint32_t f2ord(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float ord2f(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// B row of a thread's accumulator pair p (its first half): pairs 2h and 2h + 1
// are rows 4 tn .. 4 tn + 3 of half h.
__device__ __forceinline__ int gt_col(int p) { return (p >> 1) * GT_BN + (threadIdx.x & 31) * 4 + (p & 1) * 2; }

// acc[i][p] = dot(A row 8*(t/32)+i, B rows b0 + gt_col(p), + 1) over K = dp; rows
// past the end (arow -1, or from b1 on) read 0.  arow must be visible to all
// threads (shared memory) before the call.
// RAGGED: A rows are filled from the front and often short of 64, B rows of a tile's:
// warps without A rows multiply nothing, nor does any warp for a half of B past b1
// (whose acc is then 0).  Lists of ~390 rows, 20 queries of a batch each: 37 % of all
// products were padding; the scan took 263 us, 241 with this.  Where tiles are full its
// second body costs registers (k-means assignment: 92 us without, 99 with).
template <int H, bool RAGGED = false>
__device__ __forceinline__ void gt_tile(GemmTileSmem<H> &s, f32x2 (&acc)[8][2 * H], const float *__restrict__ A,
                                        const int64_t *arow, int64_t lda, const float *__restrict__ B, int64_t b0,
                                        int64_t b1, int64_t ldb, int dp) {
    const int t = threadIdx.x;
    const int tm = t >> 5, tn = t & 31;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int p = 0; p < 2 * H; ++p) acc[i][p] = 0ull;
    const int nk = dp / GT_BK;
    // this thread's float4 of each slice: row t / 4 of A, rows t / 4 + 64 h of B, k 4 (t % 4) ..
    const int r = t >> 2, k4 = t & 3;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int64_t ar = arow[r];
    const bool work = !RAGGED || arow[tm * 8] >= 0;
    const bool both = !RAGGED || H == 1 || b0 + GT_BN < b1;
    const float *ap = A + (ar >= 0 ? ar : 0) * lda + 4 * k4;
    const float *bp = B + (b0 + r) * ldb + 4 * k4;
    float4 ra, rb[2 * H];
    auto load = [&](int k0) {
        ra = ar >= 0 ? *reinterpret_cast<const float4 *>(ap + k0) : zero;
#pragma unroll
        for (int h = 0; h < 2 * H; ++h)
            rb[h] = b0 + r + 64 * h < b1 ? *reinterpret_cast<const float4 *>(bp + (int64_t)64 * h * ldb + k0) : zero;
    };
    auto store = [&](int buf) {
        s.As[buf][4 * k4 + 0][r] = make_float2(ra.x, ra.x);
        s.As[buf][4 * k4 + 1][r] = make_float2(ra.y, ra.y);
        s.As[buf][4 * k4 + 2][r] = make_float2(ra.z, ra.z);
        s.As[buf][4 * k4 + 3][r] = make_float2(ra.w, ra.w);
#pragma unroll
        for (int h = 0; h < 2 * H; ++h) {
            s.Bs[buf][4 * k4 + 0][r + 64 * h] = rb[h].x;
            s.Bs[buf][4 * k4 + 1][r + 64 * h] = rb[h].y;
            s.Bs[buf][4 * k4 + 2][r + 64 * h] = rb[h].z;
            s.Bs[buf][4 * k4 + 3][r + 64 * h] = rb[h].w;
        }
    };
    load(0);
    store(0);
    __syncthreads();
    for (int kc = 0; kc < nk; ++kc) {
        const int cur = kc & 1;
        if (kc + 1 < nk) load((kc + 1) * GT_BK);
        auto slice = [&](auto HC) {  // the first HC halves
            constexpr int HN = decltype(HC)::value;
#pragma unroll
            for (int kk = 0; kk < GT_BK; ++kk) {
                f32x2 av[8], bv[2 * HN];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&s.As[cur][kk][tm * 8 + 2 * i]);
                    av[2 * i] = x.x;
                    av[2 * i + 1] = x.y;
                }
#pragma unroll
                for (int h = 0; h < HN; ++h) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&s.Bs[cur][kk][h * GT_BN + tn * 4]);
                    bv[2 * h] = x.x;
                    bv[2 * h + 1] = x.y;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int p = 0; p < 2 * HN; ++p) acc[i][p] = fma2(av[i], bv[p], acc[i][p]);
            }
        };
        if (work && both) slice(std::integral_constant<int, H>());
        else if (work) slice(std::integral_constant<int, 1>());
        if (kc + 1 < nk) store(cur ^ 1);
        __syncthreads();
    }
}

}  // namespace gn
