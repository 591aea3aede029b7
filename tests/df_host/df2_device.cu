// Device build of the packed df64 operations (df64.cuh's df2) and of the df64 and f32c
// pairs, for tests/test_df2_gpu.py.  Built twice: with the packed FP32 instructions,
// as the library is, and with DDD_F2_PLAIN, the same source on scalar ones.
#include <cuda_runtime.h>

#include <cstdint>

#include "pair_df.cuh"

using namespace ddd;

namespace {

__device__ bool same(df64 a, df64 b) {
  return __float_as_int(a.hi) == __float_as_int(b.hi) && __float_as_int(a.lo) == __float_as_int(b.lo);
}

constexpr int kOps = 19;

// v: 6 doubles per case, three operands for each lane; bad[op] counts lanes that differ
// from the scalar operation.
__global__ void ops(const double* __restrict__ v, int64_t n, unsigned long long* __restrict__ bad) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* w = v + 6 * i;
  const df64 a = df_from_double(w[0]), b = df_from_double(w[1]), g = df_from_double(w[2]);
  const df64 c = df_from_double(w[3]), d = df_from_double(w[4]), h = df_from_double(w[5]);
  const df64 pa = a.hi < 0.0f ? -a : a, pc = c.hi < 0.0f ? -c : c;
  const df2 P = df2_make(a, c), Q = df2_make(b, d), G = df2_make(g, h), PP = df2_make(pa, pc);
  auto check = [&](int op, df2 r, df64 x, df64 y) {
    const int k = !same(df2_x(r), x) + !same(df2_y(r), y);
    if (k) atomicAdd(&bad[op], (unsigned long long)k);
  };
  check(0, P + Q, a + b, c + d);
  check(1, P - Q, a - b, c - d);
  check(2, P * Q, a * b, c * d);
  check(3, P / Q, a / b, c / d);
  check(4, df_recip(P), df_recip(a), df_recip(c));
  check(5, df_sqrt(PP), df_sqrt(pa), df_sqrt(pc));
  check(6, df_log(PP), df_log(pa), df_log(pc));
  check(7, df_atan(P), df_atan(a), df_atan(c));
  check(8, P + Q.hi, a + b.hi, c + d.hi);
  check(9, P - Q.hi, a - b.hi, c - d.hi);
  check(10, P * Q.hi, a * b.hi, c * d.hi);
  // Compositions: what a compiler could fuse across operations.
  check(11, P * Q + G, a * b + g, c * d + h);
  check(12, G - P * Q, g - a * b, h - c * d);
  check(13, P * Q * G, a * b * g, c * d * h);
  check(14, P * Q - P * G, a * b - a * g, c * d - c * h);
  check(15, (P + Q) * (P - G), (a + b) * (a - g), (c + d) * (c - h));
  check(16, df_scale(P, 2.0f) * Q + P * Q.hi, df_scale(a, 2.0f) * b + a * b.hi, df_scale(c, 2.0f) * d + c * d.hi);
  check(17, df_sqrt(PP * PP + Q * Q), df_sqrt(pa * pa + b * b), df_sqrt(pc * pc + d * d));
  check(18, P * df_log(PP) - Q / P, a * df_log(pa) - b / a, c * df_log(pc) - d / c);
}

__device__ DV3 dv3(const double* v) { return {df_from_double(v[0]), df_from_double(v[1]), df_from_double(v[2])}; }

// Pair q: rows 2 q and 2 q + 1 of segs (13 doubles: n1, n2, b, t, 1/l); its twelve
// components as (hi, lo).
template <int FORM>
__global__ void pairs(KConstsDF K, KConstsF KF, const double* __restrict__ segs, int64_t n, float* __restrict__ out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= n) return;
  const double *a = segs + 26 * q, *b = a + 13;
  const DV3 n11 = dv3(a), n12 = dv3(a + 3), b1 = dv3(a + 6), t1 = dv3(a + 9);
  const DV3 n21 = dv3(b), n22 = dv3(b + 3), b2 = dv3(b + 6), t2 = dv3(b + 9);
  const df64 t1N = df_from_double(a[12]), t2N = df_from_double(b[12]), c = dot(t1, t2);
  DV3 F[4];
  if (FORM == 0)
    general_pair_df<true, true>(K, b1, n11, n12, t1, t1N, b2, n21, n22, t2, t2N, c, F[0], F[1], F[2], F[3]);
  else
    general_pair_mixed<true, true, true>(K, KF, f3(b1), n11, n12, t1, t1N.hi, f3(b2), n21, n22, t2, t2N.hi, c, F[0],
                                         F[1], F[2], F[3]);
  for (int k = 0; k < 4; ++k) {
    const df64 v[3] = {F[k].x, F[k].y, F[k].z};
    for (int x = 0; x < 3; ++x) {
      out[24 * q + 6 * k + 2 * x] = v[x].hi;
      out[24 * q + 6 * k + 2 * x + 1] = v[x].lo;
    }
  }
}

struct Dev {
  void* p = nullptr;
  explicit Dev(size_t bytes) { ok = cudaMalloc(&p, bytes) == cudaSuccess; }
  ~Dev() { cudaFree(p); }
  bool ok;
};

}  // namespace

extern "C" int df2_ops() { return kOps; }

extern "C" int df2_compare(const double* v, int64_t n, int64_t* bad) {
  Dev dv(48 * n), db(8 * kOps);
  if (!dv.ok || !db.ok || cudaMemcpy(dv.p, v, 48 * n, cudaMemcpyHostToDevice) != cudaSuccess) return 1;
  if (cudaMemset(db.p, 0, 8 * kOps) != cudaSuccess) return 1;
  ops<<<(unsigned)((n + 127) / 128), 128>>>((const double*)dv.p, n, (unsigned long long*)db.p);
  return cudaMemcpy(bad, db.p, 8 * kOps, cudaMemcpyDeviceToHost) != cudaSuccess;
}

// k: aSq, mu4pi, mu8pi, mu4pinu; form 0 df64, 1 f32c; out: 24 floats per pair.
extern "C" int df2_pairs(int form, const double* k, const double* segs, int64_t n, float* out) {
  const double mu8piaSq = k[0] * k[2], mu4pinuaSq = k[0] * k[3];
  auto split = [](double x) {
    const float hi = (float)x;
    return df64{hi, (float)(x - (double)hi)};
  };
  const KConstsDF K{split(k[0]), split(k[1]), split(k[3]), split(mu8piaSq), split(mu4pinuaSq)};
  const KConstsF KF{(float)k[1], (float)k[3], (float)mu8piaSq, (float)mu4pinuaSq};
  Dev ds(208 * n), dout(96 * n);
  if (!ds.ok || !dout.ok || cudaMemcpy(ds.p, segs, 208 * n, cudaMemcpyHostToDevice) != cudaSuccess) return 1;
  const unsigned grid = (unsigned)((n + 127) / 128);
  if (form == 0)
    pairs<0><<<grid, 128>>>(K, KF, (const double*)ds.p, n, (float*)dout.p);
  else
    pairs<1><<<grid, 128>>>(K, KF, (const double*)ds.p, n, (float*)dout.p);
  return cudaMemcpy(out, dout.p, 96 * n, cudaMemcpyDeviceToHost) != cudaSuccess;
}
