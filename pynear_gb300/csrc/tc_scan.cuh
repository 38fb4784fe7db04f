// tc_scan.cuh — launcher interface of the tensor-core candidate stage.
#pragma once

#include "index.cuh"

namespace gn {

// One work unit of the IVF scans (tc_ivf.cu): query rows [a0, a0 + na) against rows
// [r0, r1), whose scores go to the query rows' score segments.
struct TcUnit {
    int64_t a0;
    int64_t r0;
    int64_t r1;
    int64_t rbase;  // first row of the list the unit belongs to
    int64_t xrow;   // IVF list scan, tiled row layout: the padded row of r0 (a multiple of 128)
    int32_t na;
};

// Operand form of a scan: BF16 rows, FP8 E4M3 rows with one FP32 scale each, or
// bits as E4M3 +1 / -1 (exact Hamming).
enum TcMode : int { TC_BF16 = 0, TC_FP8 = 1, TC_SIGN = 2 };

// Slack that makes a bound on scores one on exact distances (q2: |q|^2 per query,
// null: none; xmax2: the largest |x|^2, float bits).
struct TcSlack {
    const float *q2 = nullptr;
    const uint32_t *xmax2 = nullptr;
    int *overflow = nullptr;
    float cross = 0.f, norm = 0.f, rel = 0.f;
};

struct TcLaunch {
    int mode = TC_BF16;
    const void *A = nullptr;       // nq query rows of K elements, K-major (a_rows of them allocated, >= 128)
    int64_t nq = 0, a_rows = 0;
    const void *B = nullptr;       // n database rows (b_rows allocated, >= 256)
    int64_t n = 0, b_rows = 0;
    int K = 0;                     // elements: multiple of 64 (BF16) or 128 (FP8)
    int nbits = 0;                 // TC_SIGN: bits per row
    const float *bnorm = nullptr;  // |B row|^2, FP32, whole 256-row tiles, NaN past n (not TC_SIGN)
    const float *ascale = nullptr, *bscale = nullptr;  // TC_FP8 (bscale: whole tiles)
    const float *pnorm = nullptr, *pscale = nullptr;   // the same of the pilot's rows (tc_pilot_values)
    uint64_t *part = nullptr;      // per query slot_keys keys: its candidate list ...
    int *qcount = nullptr;         // ... and its length (the S best keys are among them)
    int *err = nullptr;            // device error word (0 = ok)
    int S = 40;                    // best keys wanted per query, <= 96
    int bound_rank = 0;            // rows that must reach the pilot's bound (0: S) ...
    TcSlack slack;                 // ... and how far it is raised
    int *overflow = nullptr;       // set where a list had to be cut to its S best (null: that is what is wanted)
};

// Launch shape for nq queries over n rows.
struct TcPlan {
    int nchunks = 1;                                       // database chunks
    int keep = 0;                                          // entries of a buffer that a unit hands over at most
    int64_t slot_keys = 0;                                 // room of a query's candidate list
    int pilot_chunks = 0, pilot_stride = 1;                // 0: no pilot
    int64_t pilot_tiles = 0;
};

// Device scratch of a scan, kept by the index.
struct TcScratch {
    DBuf qbound, cand, gmin;
};

// Kernel arguments.
struct TcScanArgs {
    int64_t nq, n, ntiles;
    int nk, kblk, stages, resident, nchunks, S, keep, nbits;
    const float *bnorm, *ascale, *bscale;
    int64_t slot_keys;
    uint64_t *part;
    int *qcount;
    uint32_t *qbound;
    uint2 *cand;
    float *gmin;
    int *err;
    int *overflow;
};

int tc_pilot_stride(int64_t n);
int tc_pilot_values(const float *x, int64_t n, DBuf &out, cudaStream_t st);
TcPlan tc_plan(int mode, int K, int64_t nq, int64_t n, int S);
int tc_topk_launch(const TcLaunch &a, const TcPlan &p, TcScratch &sc, cudaStream_t st);
// Exact k-NN of a flat Hamming or L2 index on the tensor cores: whether a search
// should take it, the search on device buffers (err: device error word), and the
// end of what it keeps of the rows.  L2: *flag is a device word; where it is not 0
// once the stream gets there, the FP32 scan has to answer.
bool ham_tc_wanted(const gn_index *ix, int64_t nq, int64_t k);
int ham_tc_search(gn_index *ix, const void *d_q, int64_t nq, int k, int64_t *d_idx, int64_t *d_dist, int *err,
                  cudaStream_t st);
bool l2_tc_wanted(gn_index *ix, int64_t nq, int64_t k);
int l2_tc_search(gn_index *ix, const float *d_q, int64_t nq, int k, int64_t *d_idx, float *d_dist, int *err,
                 const int **flag, cudaStream_t st);
void flat_tc_reset(gn_index *ix);
void to_bf16_rows(const float *X, int64_t n, int d, int ldx, void *out, int K, cudaStream_t st);
void to_e4m3_rows(const float *X, int64_t n, int d, int ldx, void *out, float *scale, int K, cudaStream_t st);

}  // namespace gn
