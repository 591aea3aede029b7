// Host build of the launch plans (ddd_internal.h).
#include "ddd_internal.h"

using namespace ddd;

extern "C" {
// The row plan of a call: column blocks, steps per CTA, rows per launch.
void plan_rows(int64_t npad, int64_t nRows, int64_t limit, int64_t* out) {
  const RowPlan p = row_plan(npad, nRows);
  out[0] = p.nBlk;
  out[1] = p.m;
  out[2] = rows_per_chunk(p, nRows, limit);
}
// The chunk of a few-point stress call (evaluations), its scratch, its point limit.
void plan_sigma(int64_t nSeg, int64_t M, int64_t* out) {
  out[0] = sigma_split_chunk(nSeg, M);
  out[1] = (int64_t)sigma_split_bytes(out[0], (nSeg + 127) / 128 * 128);
  out[2] = kSigmaSplitPoints;
}
}
