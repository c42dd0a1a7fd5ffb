// scan_tc.cuh -- interface between the scan's entry points (scan.cu) and its tensor-core ranking pass (scan_tc.cu).
#pragma once
#include "common.cuh"

namespace tqb {

struct ScanTcArgs {
    const uint8_t* records; int rec_bytes;                 // MSE index: key-only records; or, Prod rows:
    const uint8_t* packed; const float* norms; const uint8_t* signs; const float* res_norms; float sign_coef;
    int64_t rows;                                          // a multiple of 16
    int dim, bits, nq;                                     // bits: of the Lloyd-Max codes
    bool proven;                                           // the merge proves its selection
    const float* cent; const float* qrot; const float* qsign;   // rotated (and, Prod, projected) queries, (nq, dim)
    // workspace
    uint8_t* images; float* gmax; float* thr;
    int* count; float* buf_s; int* buf_i; int cap;         // candidates of a query: count[q], then buf_*[q * cap ..]
    uint32_t* limits;                                      // largest |norm| and sign magnitude of the rows (float bits), 1 = a wait expired
    float2* qsum;                                          // sums of the magnitudes of a query's two (scaled) columns
    int* error;
    // plan (gx: CTAs of a query block in the sampling launch)
    int cols, blocks, gx, stride, ksel, rank, flushes, tiles_per_flush, groups;
};
struct ScanTcPlan { size_t off_images, off_gmax, off_thr, off_count, off_limits, off_qsum, off_s, off_i, total; int cap, cols, blocks, gx; };

constexpr int SCAN_TC_MIN_QUERIES = 9;                     // MSE calls of fewer queries never take the pass
// Workspace and shape of the pass (nothing for such calls); independent of the number of rows.
ScanTcPlan scan_tc_plan(int nq, int dim, bool prod, int ksel);
// Whether the pass is taken for this call (the reasons are in scan_tc.cu).  `proven`: its selection has to be proven, see below.
bool scan_tc_wanted(int nq, int64_t rows, int dim, int bits, bool prod, int ksel, bool proven);
// Candidates of every query into its buffer: everything not below a bound (thr) of the ksel-th best approximate score.  A query
// with count[q] > cap has overflowed (more rows tie with the bound than the buffer holds, or a wait expired): its buffer is
// not used.
int scan_tc_run(ScanTcArgs a, const ScanTcPlan& pl, uint8_t* ws, cudaStream_t st);

// Largest difference between a row's approximate score (in its query's scale) and its float32 score, for rows whose norms and
// sign magnitudes are at most those in `limits`: fp16 rounds the centroids, the queries and the sign magnitude by 2^-11 of
// their size or 2^-25, which the products carry into the sum of their magnitudes; 6 % more for second orders, the float32
// sums of both sides and the tensor core's accumulator (dim 2^-24, and 2^-22 for each of its 16 steps at most).
// cmax: largest |centroid| in the operand's scale.
__device__ __forceinline__ float scan_tc_error(const uint32_t* limits, float2 qsum, float cmax, int dim) {
    const float norm = __uint_as_float(limits[0]), sign = __uint_as_float(limits[1]);
    const float rel = 1.06f / 1024.0f * fmaf(cmax, qsum.x, sign * qsum.y);
    const float sub = 5.9604645e-8f * (qsum.x + qsum.y + (float)dim * (cmax + sign + 1.0f));
    return norm * (rel + sub);
}

}  // namespace tqb
