// voronoi.cu — headless Voronoi raster: every pixel of a w×h grid gets the
// index of its nearest seed (exact 1-NN in 2-D, L2), optionally its distance
// and an RGBA colour from a palette, written to device or host buffers.
//
// The reference computes the same raster by building a pixel grid on the host
// (pixel (r, c) = (xs[c], ys[r]), xs/ys = linspace(0, 1)) and running one
// search1NN of all pixels against the seeds (demo/voronoi.py:93-110).  Here the
// grid is never materialised: the kernel reads the two coordinate vectors.
//
// Answer per pixel: the lexicographic minimum of (sqrt(rn(rn(dx²) + rn(dy²))),
// seed index), dx = px − sx, dy = py − sy, the flat L2 kernel's arithmetic for
// d = 2.  Seeds are offered in index order; a squared sum below the best one
// is needed to win (sqrt is monotone), so the sqrt is rarely taken.
//
// Seeds that cannot win are left out by tiles of pixels, in two levels: a
// block's tile (128 x 64 pixels, 32 x 32 where that leaves SMs idle), then a
// warp's 16 x 8.  For a tile with coordinates in [x0, x1] x [y0, y1], a seed's
// |dx| lies between the rounded distances from sx to the interval's nearest and
// farthest end, because rounding is monotone, and so are the rounded square,
// sum and root: with lb / ub the same arithmetic on those ends,
//     lb(seed) <= its squared sum at every pixel of the tile <= ub(seed)
// holds exactly, without a margin.  A seed with sqrt(lb) > sqrt(min ub) is
// strictly farther than another one everywhere in the tile; equal roots are
// kept, so ties still go to the lower index.  NaN pixels keep id 0 and +inf
// whatever is left out, NaN seeds never win, and an infinite pixel coordinate
// makes min ub infinite, which keeps every seed.
//
// A handful of seeds is not worth the bounds: voronoi_few_kernel evaluates all of
// them for four neighbouring pixels a thread.
//
// Block list: up to VR_CAP surviving seeds in shared memory; where more
// survive (seeds crowded together), the warps read all seeds instead.  A warp
// collects its own survivors VR_WCAP at a time and evaluates four seeds for
// its four neighbouring pixels per thread in packed FP32 (two results an
// instruction: the loop is bound by issue slots).  3840 x 2160, 4,096 seeds:
// 5.12 ms evaluating every pair, 0.068 ms with the tiles (66 MB of ids and
// colours out: 0.010 ms of HBM time; what is left is the two levels of bounds).
#include <cmath>

#include "f32x2.cuh"
#include "index.cuh"

namespace gn {

constexpr int VR_NT = 256;    // threads per block
constexpr int VR_WARPS = VR_NT / 32;
constexpr int VR_CAP = 1024;  // seeds in a block's list
constexpr int VR_WCAP = 64;   // seeds a warp collects before it evaluates them (a multiple of 32)
constexpr int VR_SW = 16, VR_SH = 8;  // a warp's pixels: four neighbours per thread

// Smallest and largest squared sum of a seed over [x0, x1] x [y0, y1].
__device__ __forceinline__ void vr_bounds(float2 s, float x0, float x1, float y0, float y1, float &lb, float &ub) {
    const float ax = __fsub_rn(x0, s.x), bx = __fsub_rn(x1, s.x), ay = __fsub_rn(y0, s.y), by = __fsub_rn(y1, s.y);
    const float fx = fmaxf(fabsf(ax), fabsf(bx)), fy = fmaxf(fabsf(ay), fabsf(by));
    const float nx = fmaxf(fmaxf(ax, -bx), 0.f), ny = fmaxf(fmaxf(ay, -by), 0.f);
    lb = __fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny));
    ub = __fadd_rn(__fmul_rn(fx, fx), __fmul_rn(fy, fy));
}

// Four neighbouring pixels of a row and the nearest seed so far of each.
struct VrQuad {
    f32x2 px01, px23;
    float py, bs[4], br[4];
    int bi[4];
    __device__ __forceinline__ void start(const float (&px)[4], float y) {
        px01 = pack2(px[0], px[1]);
        px23 = pack2(px[2], px[3]);
        py = y;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            bs[p] = INFINITY;
            br[p] = INFINITY;
            bi[p] = 0;
        }
    }
    // offer seed `idx` with squared sum s to pixel p (seed order is kept)
    __device__ __forceinline__ void offer(int p, float s, int idx) {
        if (s < bs[p]) {
            const float r = __fsqrt_rn(s);
            if (r < br[p]) {  // strictly nearer: equal distances keep the lower index
                bs[p] = s;
                br[p] = r;
                bi[p] = idx;
            }
        }
    }
    // the four pixels' squared sums
    __device__ __forceinline__ void sums(float2 s, float (&o)[4]) const {
        const float dy = __fsub_rn(py, s.y);
        const f32x2 dy2 = dup2(__fmul_rn(dy, dy)), nx = dup2(-s.x);
        const f32x2 d01 = add2(px01, nx), d23 = add2(px23, nx);
        float d0, d1, d2, d3;
        unpack2(d01, d0, d1);
        unpack2(d23, d2, d3);
        // scalar products: a packed product and sum came out fused (one rounding
        // instead of the two of the reference's arithmetic)
        unpack2(add2(pack2(__fmul_rn(d0, d0), __fmul_rn(d1, d1)), dy2), o[0], o[1]);
        unpack2(add2(pack2(__fmul_rn(d2, d2), __fmul_rn(d3, d3)), dy2), o[2], o[3]);
    }
    __device__ __forceinline__ void seed(float2 s, int idx) {
        float o[4];
        sums(s, o);
#pragma unroll
        for (int p = 0; p < 4; ++p) offer(p, o[p], idx);
    }
    // the outputs of pixels pc .. pc + 3 (those below w) of row pr
    __device__ __forceinline__ void store(int pr, int pc, int w, int32_t *__restrict__ ids, float *__restrict__ dist,
                                          const uchar4 *__restrict__ palette, int npal,
                                          uchar4 *__restrict__ rgba) const {
        const int64_t off = (int64_t)pr * w + pc;
        const int here = w - pc;
        uchar4 col[4];
        if (rgba) {
#pragma unroll
            for (int p = 0; p < 4; ++p) col[p] = palette[bi[p] < npal ? bi[p] : bi[p] % npal];
        }
        // whole 16-byte stores where the row starts allow them
        const bool vec = here >= 4 && (w & 3) == 0;
        if (ids) {
            if (vec && ((uintptr_t)ids & 15) == 0) {
                *reinterpret_cast<int4 *>(ids + off) = make_int4(bi[0], bi[1], bi[2], bi[3]);
            } else {
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (p < here) ids[off + p] = bi[p];
            }
        }
        if (dist) {
            if (vec && ((uintptr_t)dist & 15) == 0) {
                *reinterpret_cast<float4 *>(dist + off) = make_float4(br[0], br[1], br[2], br[3]);
            } else {
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (p < here) dist[off + p] = br[p];
            }
        }
        if (rgba) {
            if (vec && ((uintptr_t)rgba & 15) == 0) {
                uint4 v;
                v.x = *reinterpret_cast<unsigned *>(&col[0]);
                v.y = *reinterpret_cast<unsigned *>(&col[1]);
                v.z = *reinterpret_cast<unsigned *>(&col[2]);
                v.w = *reinterpret_cast<unsigned *>(&col[3]);
                *reinterpret_cast<uint4 *>(rgba + off) = v;
            } else {
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (p < here) rgba[off + p] = col[p];
            }
        }
    }
};

// Block tile: TX x TY warp tiles.
template <int TX, int TY>
__global__ void __launch_bounds__(VR_NT) voronoi_kernel(const float2 *__restrict__ seeds, int ns,
                                                        const float *__restrict__ xs, const float *__restrict__ ys,
                                                        int w, int h, int tiles_y, int32_t *__restrict__ ids,
                                                        float *__restrict__ dist,
                                                        const uchar4 *__restrict__ palette, int npal,
                                                        uchar4 *__restrict__ rgba) {
    __shared__ float2 bxy[VR_CAP];
    __shared__ int bid[VR_CAP];
    __shared__ float2 wxy[VR_WARPS][VR_WCAP + 32];
    __shared__ int wid[VR_WARPS][VR_WCAP + 32];
    __shared__ float red[5][VR_WARPS];
    __shared__ int wcount[VR_WARPS];
    constexpr float INF = INFINITY;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int ty = blockIdx.y; ty < tiles_y; ty += gridDim.y) {
        const int c0 = blockIdx.x * TX * VR_SW, r0 = ty * TY * VR_SH;
        const int nc = min(TX * VR_SW, w - c0), nr = min(TY * VR_SH, h - r0);
        // the tile's coordinate ranges (NaN coordinates drop out of the minima)
        float x0 = INF, x1 = -INF, y0 = INF, y1 = -INF;
        for (int i = t; i < nc; i += VR_NT) {
            x0 = fminf(x0, xs[c0 + i]);
            x1 = fmaxf(x1, xs[c0 + i]);
        }
        for (int i = t; i < nr; i += VR_NT) {
            y0 = fminf(y0, ys[r0 + i]);
            y1 = fmaxf(y1, ys[r0 + i]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
            y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
            y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
        }
        __syncthreads();  // the previous tile is done with the lists
        if (lane == 0) {
            red[0][warp] = x0;
            red[1][warp] = x1;
            red[2][warp] = y0;
            red[3][warp] = y1;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < VR_WARPS; ++i) {
            x0 = fminf(x0, red[0][i]);
            x1 = fmaxf(x1, red[1][i]);
            y0 = fminf(y0, red[2][i]);
            y1 = fmaxf(y1, red[3][i]);
        }
        // some seed is within `u` of every pixel
        float u = INF, lb, ub;
        for (int j = t; j < ns; j += VR_NT) {
            vr_bounds(seeds[j], x0, x1, y0, y1, lb, ub);
            u = fminf(u, ub);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) u = fminf(u, __shfl_xor_sync(0xffffffffu, u, o));
        if (lane == 0) red[4][warp] = u;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < VR_WARPS; ++i) u = fminf(u, red[4][i]);
        u = __fsqrt_rn(u);
        // the block's list, in index order
        int m = 0;
        for (int j0 = 0; j0 < ns && m <= VR_CAP; j0 += VR_NT) {
            const int j = j0 + t;
            float2 s = make_float2(0.f, 0.f);
            bool keep = false;
            if (j < ns) {
                s = seeds[j];
                vr_bounds(s, x0, x1, y0, y1, lb, ub);
                keep = __fsqrt_rn(lb) <= u;
            }
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) wcount[warp] = __popc(mask);
            __syncthreads();
            int before = m, all = 0;
#pragma unroll
            for (int i = 0; i < VR_WARPS; ++i) {
                const int cnt = wcount[i];
                if (i < warp) before += cnt;
                all += cnt;
            }
            const int at = before + __popc(mask & ((1u << lane) - 1));
            if (keep && at < VR_CAP) {
                bxy[at] = s;
                bid[at] = j;
            }
            m += all;
            __syncthreads();
        }
        const bool listed = m <= VR_CAP;  // else: too many, read the seeds themselves
        const int nsrc = listed ? m : ns;

        for (int wt = warp; wt < TX * TY; wt += VR_WARPS) {
            const int oc = (wt % TX) * VR_SW, orow = (wt / TX) * VR_SH;
            if (oc >= nc || orow >= nr) continue;
            // (unsigned: the last tile's pixels may lie past the largest int)
            const unsigned pc = (unsigned)(c0 + oc) + (lane & 3) * 4, pr = (unsigned)(r0 + orow) + (lane >> 2);
            const float py = ys[min(pr, (unsigned)h - 1)];
            float px[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) px[p] = xs[min(pc + p, (unsigned)w - 1)];
            float a0 = fminf(fminf(px[0], px[1]), fminf(px[2], px[3])), b0 = py;
            float a1 = fmaxf(fmaxf(px[0], px[1]), fmaxf(px[2], px[3])), b1 = py;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                a0 = fminf(a0, __shfl_xor_sync(0xffffffffu, a0, o));
                a1 = fmaxf(a1, __shfl_xor_sync(0xffffffffu, a1, o));
            }
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                b0 = fminf(b0, __shfl_xor_sync(0xffffffffu, b0, o));
                b1 = fmaxf(b1, __shfl_xor_sync(0xffffffffu, b1, o));
            }
            float wu = INF;
            for (int j = lane; j < nsrc; j += 32) {
                vr_bounds(listed ? bxy[j] : seeds[j], a0, a1, b0, b1, lb, ub);
                wu = fminf(wu, ub);
            }
            wu = __fsqrt_rn(__uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(wu))));

            VrQuad px4;
            px4.start(px, py);
            float2 *lxy = wxy[warp];
            int *lid = wid[warp];
            auto evaluate = [&](int cnt) {
                int j = 0;
                for (; j + 4 <= cnt; j += 4) {
                    float s0[4], s1[4], s2[4], s3[4];
                    px4.sums(lxy[j], s0);
                    px4.sums(lxy[j + 1], s1);
                    px4.sums(lxy[j + 2], s2);
                    px4.sums(lxy[j + 3], s3);
#pragma unroll
                    for (int p = 0; p < 4; ++p)
                        if (fminf(fminf(s0[p], s1[p]), fminf(s2[p], s3[p])) < px4.bs[p]) {
                            px4.offer(p, s0[p], lid[j]);
                            px4.offer(p, s1[p], lid[j + 1]);
                            px4.offer(p, s2[p], lid[j + 2]);
                            px4.offer(p, s3[p], lid[j + 3]);
                        }
                }
                for (; j < cnt; ++j) px4.seed(lxy[j], lid[j]);
            };
            int cnt = 0;
            for (int j0 = 0; j0 < nsrc; j0 += 32) {
                const int j = j0 + lane;
                float2 s = make_float2(0.f, 0.f);
                bool keep = false;
                if (j < nsrc) {
                    s = listed ? bxy[j] : seeds[j];
                    vr_bounds(s, a0, a1, b0, b1, lb, ub);
                    keep = __fsqrt_rn(lb) <= wu;
                }
                const unsigned mask = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const int at = cnt + __popc(mask & ((1u << lane) - 1));
                    lxy[at] = s;
                    lid[at] = listed ? bid[j] : j;
                }
                cnt += __popc(mask);
                if (cnt >= VR_WCAP) {
                    __syncwarp();
                    evaluate(cnt);
                    __syncwarp();
                    cnt = 0;
                }
            }
            __syncwarp();
            evaluate(cnt);
            __syncwarp();

            if (pr < (unsigned)h && pc < (unsigned)w)
                px4.store((int)pr, (int)pc, w, ids, dist, palette, npal, rgba);
        }
    }
}

// Few seeds: every seed for every pixel, a warp to 128 pixels of a row.
constexpr int VR_FROWS = 8;
__global__ void __launch_bounds__(32 * VR_FROWS)
    voronoi_few_kernel(const float2 *__restrict__ seeds, int ns, const float *__restrict__ xs,
                       const float *__restrict__ ys, int w, int h, int32_t *__restrict__ ids,
                       float *__restrict__ dist, const uchar4 *__restrict__ palette, int npal,
                       uchar4 *__restrict__ rgba) {
    const int64_t pc = (int64_t)blockIdx.x * 128 + (threadIdx.x & 31) * 4;
    if (pc >= w) return;
    float px[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) px[p] = xs[min(pc + p, (int64_t)w - 1)];
    for (int64_t pr = (int64_t)blockIdx.y * VR_FROWS + (threadIdx.x >> 5); pr < h; pr += (int64_t)gridDim.y * VR_FROWS) {
        VrQuad px4;
        px4.start(px, ys[pr]);
        for (int j = 0; j < ns; ++j) px4.seed(__ldg(seeds + j), j);
        px4.store((int)pr, (int)pc, w, ids, dist, palette, npal, rgba);
    }
}

static int voronoi_check(int64_t ns, int64_t w, int64_t h, const void *seeds, const void *xs, const void *ys,
                         const void *ids, const void *dist, const void *palette, int64_t npal, const void *rgba) {
    if (ns <= 0) return fail(GN_ERR_EMPTY, "voronoi raster needs at least one seed");
    if (ns > 0x7fffffffLL) return fail(GN_ERR_INVALID, "too many seeds");
    if (w <= 0 || h <= 0 || w > 0x7fffffffLL || h > 0x7fffffffLL)
        return fail(GN_ERR_INVALID, "raster width and height must be positive");
    if (!seeds || !xs || !ys) return fail(GN_ERR_INVALID, "NULL pointer argument");
    if (!ids && !dist && !rgba) return fail(GN_ERR_INVALID, "no output requested");
    if (rgba && (!palette || npal <= 0 || npal > 0x7fffffffLL))
        return fail(GN_ERR_INVALID, "an RGBA output needs a non-empty palette");
    return GN_OK;
}

static int voronoi_launch(const float *seeds, int64_t ns, const float *xs, const float *ys, int64_t w, int64_t h,
                          int32_t *ids, float *dist, const uint8_t *palette, int64_t npal, uint8_t *rgba,
                          cudaStream_t st) {
    if ((reinterpret_cast<uintptr_t>(seeds) & 7) || (reinterpret_cast<uintptr_t>(palette) & 3) ||
        (reinterpret_cast<uintptr_t>(rgba) & 3))
        return fail(GN_ERR_INVALID, "seeds must be 8-byte aligned, palette and RGBA output 4-byte aligned");
    auto launch = [&](auto kern, int tw, int th) {
        const int64_t tiles_y = ceil_div(h, th);
        dim3 grid((unsigned)ceil_div(w, tw), (unsigned)std::min<int64_t>(tiles_y, 65535));
        kern<<<grid, VR_NT, 0, st>>>(reinterpret_cast<const float2 *>(seeds), (int)ns, xs, ys, (int)w, (int)h,
                                     (int)tiles_y, ids, dist, reinterpret_cast<const uchar4 *>(palette), (int)npal,
                                     reinterpret_cast<uchar4 *>(rgba));
    };
    // Few seeds are cheaper without the tiles' bounds, the more so where there are few
    // pixels for a block's bounds to serve.  In us, tiles / all seeds: 1377 x 466 with 1, 8
    // and 16 seeds 9.1 / 3.6, 9.1 / 5.5, 9.1 / 7.3; 1920 x 1080 15.3 / 6.5, 15.5 / 11.3,
    // 15.5 / 15.9; 3840 x 2160 37 / 20, 38 / 37, 38 / 54; 7680 x 4320 with 1, 4 and 8 seeds 129 /
    // 77, 130 / 105, 130 / 141; 256 x 256 with 8 and 16 4.0 / 3.6, 4.6 / 5.4.
    const int64_t pixels = w * h;
    const int few = pixels < (1 << 18) ? 9 : pixels < (1 << 22) ? 16 : pixels < (1 << 24) ? 8 : 6;
    if (ns <= few) {
        const dim3 grid((unsigned)ceil_div(w, 128), (unsigned)std::min<int64_t>(ceil_div(h, VR_FROWS), 65535));
        voronoi_few_kernel<<<grid, 32 * VR_FROWS, 0, st>>>(
            reinterpret_cast<const float2 *>(seeds), (int)ns, xs, ys, (int)w, (int)h, ids, dist,
            reinterpret_cast<const uchar4 *>(palette), (int)npal, reinterpret_cast<uchar4 *>(rgba));
        GN_CUDA_TRY(cudaGetLastError());
        return GN_OK;
    }
    // large tiles share one pass over the seeds among 64 warp tiles; small ones
    // where large ones would not give every SM two blocks
    if (ceil_div(w, 8 * VR_SW) * ceil_div(h, 8 * VR_SH) >= 2 * dev_info().num_sms)
        launch(voronoi_kernel<8, 8>, 8 * VR_SW, 8 * VR_SH);
    else
        launch(voronoi_kernel<2, 4>, 2 * VR_SW, 4 * VR_SH);
    GN_CUDA_TRY(cudaGetLastError());
    return GN_OK;
}

}  // namespace gn

using namespace gn;

extern "C" int gn_voronoi_raster_device(const float *d_seeds, int64_t n_seeds, const float *d_xs, int64_t width,
                                        const float *d_ys, int64_t height, int32_t *d_ids, float *d_dist,
                                        const uint8_t *d_palette, int64_t n_palette, uint8_t *d_rgba,
                                        void *stream) {
    GN_TRY(voronoi_check(n_seeds, width, height, d_seeds, d_xs, d_ys, d_ids, d_dist, d_palette, n_palette, d_rgba));
    return voronoi_launch(d_seeds, n_seeds, d_xs, d_ys, width, height, d_ids, d_dist, d_palette, n_palette, d_rgba,
                          (cudaStream_t)stream);
}

extern "C" int gn_voronoi_raster(const float *seeds, int64_t n_seeds, const float *xs, int64_t width,
                                 const float *ys, int64_t height, int32_t *out_ids, float *out_dist,
                                 const uint8_t *palette, int64_t n_palette, uint8_t *out_rgba) {
    GN_TRY(voronoi_check(n_seeds, width, height, seeds, xs, ys, out_ids, out_dist, palette, n_palette, out_rgba));
    // per-thread scratch, reused by later calls of the same thread
    struct Scratch {
        DBuf seeds, xs, ys, ids, dist, pal, rgba;
        cudaStream_t st = nullptr;
    };
    static thread_local Scratch S;
    if (!S.st) GN_CUDA_TRY(cudaStreamCreateWithFlags(&S.st, cudaStreamNonBlocking));
    const size_t npx = (size_t)width * height;
    GN_TRY(S.seeds.ensure((size_t)n_seeds * 8));
    GN_TRY(S.xs.ensure((size_t)width * 4));
    GN_TRY(S.ys.ensure((size_t)height * 4));
    if (out_ids) GN_TRY(S.ids.ensure(npx * 4));
    if (out_dist) GN_TRY(S.dist.ensure(npx * 4));
    if (out_rgba) {
        GN_TRY(S.pal.ensure((size_t)n_palette * 4));
        GN_TRY(S.rgba.ensure(npx * 4));
    }
    GN_CUDA_TRY(cudaMemcpyAsync(S.seeds.p, seeds, (size_t)n_seeds * 8, cudaMemcpyHostToDevice, S.st));
    GN_CUDA_TRY(cudaMemcpyAsync(S.xs.p, xs, (size_t)width * 4, cudaMemcpyHostToDevice, S.st));
    GN_CUDA_TRY(cudaMemcpyAsync(S.ys.p, ys, (size_t)height * 4, cudaMemcpyHostToDevice, S.st));
    if (out_rgba)
        GN_CUDA_TRY(cudaMemcpyAsync(S.pal.p, palette, (size_t)n_palette * 4, cudaMemcpyHostToDevice, S.st));
    GN_TRY(voronoi_launch(S.seeds.as<float>(), n_seeds, S.xs.as<float>(), S.ys.as<float>(), width, height,
                          out_ids ? S.ids.as<int32_t>() : nullptr, out_dist ? S.dist.as<float>() : nullptr,
                          out_rgba ? S.pal.as<uint8_t>() : nullptr, n_palette,
                          out_rgba ? S.rgba.as<uint8_t>() : nullptr, S.st));
    if (out_ids) GN_CUDA_TRY(cudaMemcpyAsync(out_ids, S.ids.p, npx * 4, cudaMemcpyDeviceToHost, S.st));
    if (out_dist) GN_CUDA_TRY(cudaMemcpyAsync(out_dist, S.dist.p, npx * 4, cudaMemcpyDeviceToHost, S.st));
    if (out_rgba) GN_CUDA_TRY(cudaMemcpyAsync(out_rgba, S.rgba.p, npx * 4, cudaMemcpyDeviceToHost, S.st));
    GN_CUDA_TRY(cudaStreamSynchronize(S.st));
    return GN_OK;
}
