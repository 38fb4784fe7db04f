// flat_scan.cuh — launcher interface of the exact flat scans.
#pragma once

#include "common.cuh"

namespace gn {

struct FlatScanArgs {
    int metric = M_L2;
    const void *db = nullptr;  // n rows, stride4 * 16 bytes each (zero padded)
    int64_t n = 0;
    int d = 0;                 // real dimension (floats) or bytes (Hamming)
    int stride4 = 0;           // row stride in 16-byte units
    const void *q = nullptr;   // nq rows, same layout as db
    int64_t nq = 0;
    int k = 0;
    int64_t *out_idx = nullptr;  // nq*k
    void *out_dist = nullptr;    // nq*k float32 or int64
    int *err = nullptr;          // float metrics: device error word of the scan's bounded waits
    int *status = nullptr;  // float metrics: pinned word that the last kernel copies the error word to (may be null)
    const int *only_if = nullptr;  // float metrics: device word; 0 = the results are there already, do nothing
    // filled by flat_plan
    int warps = 4, n_slices = 1, n_groups = 1;
    int64_t slice_rows = 0;
    int64_t units = 0, list_keys = 0, gbuf_keys = 0;  // float scan: CTAs, candidates per query, buffer keys
    int64_t wave_queries = 0;  // float scan: queries better scanned on their own before the others (0: none)
};

constexpr int FLAT_MAX_K_WARP = 256;
// Queries of a float search with k > 64 scanned at a time: each block of the scan has
// its lists' buffers in global memory (4 KB per query and slice), which for a whole
// batch would outgrow its results (150,000 queries, k 100: 0.61 GB beside 0.18 GB).
// That batch over 4,096 x 5 rows: 8.5 ms in one piece, 9.0 so, 10.4 at 8,192 a time.
constexpr int64_t FLAT_QBLOCK = 32768;

void flat_plan(FlatScanArgs &a);
size_t flat_part_bytes(const FlatScanArgs &a);
int flat_smem_ok(const FlatScanArgs &a);
int flat_launch(const FlatScanArgs &a, uint64_t *part, cudaStream_t st);
// Hamming with appended candidates, and the searches that keep ordered lists instead
// (flat_plan and flat_launch, as do searches in a caller's scratch).
bool ham_ordered(const FlatScanArgs &a);
void ham_plan(FlatScanArgs &a);
size_t ham_part_bytes(const FlatScanArgs &a);
int ham_launch(const FlatScanArgs &a, uint64_t *part, cudaStream_t st);
// The k nearest (k <= 256) of each query's qcount[q] candidate (distance, index)
// keys at cand + q * list_keys, nearest first, with their number where out_cnt is given.
// only_if, err, status: see FlatScanArgs.
int candidates_finish(const uint64_t *cand, const int *qcount, int64_t list_keys, int64_t nq, int k, int64_t *out_idx,
                      float *out_dist, int64_t *out_cnt, const int *only_if, cudaStream_t st,
                      const int *err = nullptr, int *status = nullptr);
int flat_preload_hamming();
int64_t next_pow2(int64_t v);
void flat_large_k_launch(const FlatScanArgs &a, int64_t q_begin, int64_t qc, uint64_t *keys, uint64_t *sorted,
                         cudaStream_t st);

}  // namespace gn
