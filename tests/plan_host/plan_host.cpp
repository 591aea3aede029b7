// Host build of the launch plans (ddd_internal.h).
#include "ddd_internal.h"

// An allocator that counts, in place of the device's.
static size_t g_allocated = 0;
extern "C" cudaError_t cudaMalloc(void** p, size_t bytes) {
  g_allocated += bytes;
  *p = &g_allocated;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void*) { return cudaSuccess; }

using namespace ddd;

extern "C" {
// The row plan of a call: column blocks, steps per CTA, rows per launch, threads.
void plan_rows(int64_t npad, int64_t nRows, int64_t limit, int64_t df64, int64_t* out) {
  const RowPlan p = row_plan(npad, nRows, df64);
  out[0] = p.nBlk;
  out[1] = p.m;
  out[2] = rows_per_chunk(p, nRows, limit);
  out[3] = p.threads;
}
// The chunk of a few-point stress call (evaluations), its scratch, its point limit.
void plan_sigma(int64_t nSeg, int64_t M, int64_t* out) {
  out[0] = sigma_split_chunk(nSeg, M);
  out[1] = (int64_t)sigma_split_bytes(out[0], (nSeg + 127) / 128 * 128);
  out[2] = kSigmaSplitPoints;
}
// Bytes that a call allocates for a store of nb tile pairs and `slots` slots of
// partial sums, and whether both fit `limit`.
void plan_store(int64_t nb, int64_t slots, int64_t limit, int64_t* out) {
  GrowBuf store, partial;
  g_allocated = 0;
  store.ensure(expand_bytes(nb));
  partial.ensure((size_t)slots * 12 * 128 * sizeof(double));
  out[0] = (int64_t)g_allocated;
  out[1] = scratch_fits(expand_bytes(nb), (size_t)slots * 12 * 128 * sizeof(double), limit);
}
}
