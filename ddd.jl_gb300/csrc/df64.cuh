// Double-float ("df64") arithmetic on the FP32 pipes: a value is hi + lo with
// |lo| <= ulp(hi)/2, about 48 significant bits.  On GB300 the FP32 pipes issue
// 64x as many operations per clock as the FP64 pipe, so df64 runs the pair
// arithmetic several times faster than native FP64 at ~2^-47 relative precision.
//
// Algorithms (published methods, restated):
//   TwoSum (Knuth), FastTwoSum (Dekker), TwoProd via FMA;
//   add / mul / div / sqrt as in Hida, Li & Bailey, "Library for double-double
//   and quad-double arithmetic" (2001): the "sloppy" or IEEE-style addition,
//   the FMA product, division by two Newton-style corrections, sqrt by one
//   Newton step on an FP32 root;
//   log: x = 2^e m, m reduced by a 64-entry table to m/c_j in [1 - 2^-7, 1 + 2^-7],
//        log(m/c_j) = 2 atanh(u), u = (m - c_j)/(m + c_j), odd series;
//   atan: |x| > 1 folded by atan(x) = pi/2 - atan(1/x), then x = c_j + reduced
//        argument with c_j = j/32, atan(x) = atan(c_j) + atan((x - c_j)/(1 + x c_j)),
//        odd series.
// Compiled with --fmad=false so the error-free transformations stay exact;
// every fused product is an explicit fmaf.
//
// Device functions under nvcc; plain inline C++ under a host compiler, so that
// the same arithmetic can be checked on a CPU against the oracle.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define DF_HD __device__ __forceinline__
#define DDD_DF_TABLE_QUAL __device__
#else
#define DF_HD inline
#define DDD_DF_TABLE_QUAL
#include <cmath>
#endif

namespace ddd {

struct float2_ {
  float x, y;
};

#include "df64_tables.h"

DF_HD float df_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return std::fmaf(a, b, c);
#endif
}
DF_HD float df_sqrtf(float a) {
#if defined(__CUDA_ARCH__)
  return __fsqrt_rn(a);
#else
  return std::sqrt(a);
#endif
}
// Approximate quotient for the first step of a df64 division (any error < 2^-20 works).
DF_HD float df_qapprox(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fdividef(a, b);
#else
  return a / b;
#endif
}
DF_HD int32_t df_bits(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_int(f);
#else
  int32_t i;
  std::memcpy(&i, &f, 4);
  return i;
#endif
}
DF_HD float df_from_bits(int32_t i) {
#if defined(__CUDA_ARCH__)
  return __int_as_float(i);
#else
  float f;
  std::memcpy(&f, &i, 4);
  return f;
#endif
}

struct df64 {
  float hi, lo;
};

DF_HD df64 two_sum(float a, float b) {
  float s = a + b;
  float bb = s - a;
  float e = (a - (s - bb)) + (b - bb);
  return {s, e};
}
DF_HD df64 fast_two_sum(float a, float b) {  // |a| >= |b|
  float s = a + b;
  float e = b - (s - a);
  return {s, e};
}
DF_HD df64 two_prod(float a, float b) {
  float p = a * b;
  float e = df_fma(a, b, -p);
  return {p, e};
}

DF_HD df64 df(float a) { return {a, 0.0f}; }
DF_HD df64 df_from_double(double d) {
  float hi = (float)d;
  float lo = (float)(d - (double)hi);
  return {hi, lo};
}
DF_HD double df_to_double(df64 a) { return (double)a.hi + (double)a.lo; }

DF_HD df64 operator-(df64 a) { return {-a.hi, -a.lo}; }

// Addition.  DDD_DF_ACCURATE_ADD selects the IEEE-style form (error relative to
// the result); the default is the "sloppy" form (error <= ~2^-47 (|a| + |b|)),
// which is as accurate as the operands themselves whenever they carry their own
// rounding error of that size — every computed df64 value does.
DF_HD df64 operator+(df64 a, df64 b) {
#ifdef DDD_DF_ACCURATE_ADD
  df64 s = two_sum(a.hi, b.hi);
  df64 t = two_sum(a.lo, b.lo);
  s.lo += t.hi;
  s = fast_two_sum(s.hi, s.lo);
  s.lo += t.lo;
  return fast_two_sum(s.hi, s.lo);
#else
  df64 s = two_sum(a.hi, b.hi);
  s.lo += a.lo + b.lo;
  return fast_two_sum(s.hi, s.lo);
#endif
}
DF_HD df64 operator-(df64 a, df64 b) { return a + (-b); }
DF_HD df64 operator+(df64 a, float b) {
  df64 s = two_sum(a.hi, b);
  s.lo += a.lo;
  return fast_two_sum(s.hi, s.lo);
}
DF_HD df64 operator-(df64 a, float b) { return a + (-b); }
DF_HD df64 operator+(float a, df64 b) { return b + a; }
DF_HD df64 operator-(float a, df64 b) { return (-b) + a; }

DF_HD df64 operator*(df64 a, df64 b) {
  df64 p = two_prod(a.hi, b.hi);
  p.lo = df_fma(a.hi, b.lo, p.lo);
  p.lo = df_fma(a.lo, b.hi, p.lo);
  return fast_two_sum(p.hi, p.lo);
}
DF_HD df64 operator*(df64 a, float b) {
  df64 p = two_prod(a.hi, b);
  p.lo = df_fma(a.lo, b, p.lo);
  return fast_two_sum(p.hi, p.lo);
}
DF_HD df64 operator*(float a, df64 b) { return b * a; }
// Exact scaling by a power of two.
DF_HD df64 df_scale(df64 a, float p2) { return {a.hi * p2, a.lo * p2}; }

DF_HD df64 operator/(df64 a, df64 b) {
  float q1 = df_qapprox(a.hi, b.hi);
  df64 r = a - b * q1;
  float q2 = df_qapprox(r.hi, b.hi);
  r = r - b * q2;
  float q3 = df_qapprox(r.hi, b.hi);
  df64 q = fast_two_sum(q1, q2);
  return q + q3;
}
DF_HD df64 df_recip(df64 b) { return df(1.0f) / b; }

DF_HD df64 df_sqrt(df64 a) {
  if (!(a.hi > 0.0f)) return {a.hi == 0.0f ? 0.0f : df_sqrtf(a.hi), 0.0f};
  float s = df_sqrtf(a.hi);
  df64 r = a - two_prod(s, s);
  float corr = df_qapprox(r.hi, 2.0f * s);
  return fast_two_sum(s, corr);
}

DF_HD bool operator>(df64 a, df64 b) { return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo); }
DF_HD bool operator<(df64 a, df64 b) { return b > a; }

// Natural logarithm, a > 0 and normal.
DF_HD df64 df_log(df64 a) {
  const int32_t bits = df_bits(a.hi);
  const int32_t e = ((bits >> 23) & 0xff) - 127;
  const int32_t j = (bits >> 17) & 63;            // top 6 mantissa bits
  const float scale = df_from_bits((127 - e) << 23);  // 2^-e, exact
  const df64 m = {a.hi * scale, a.lo * scale};        // m in [1, 2)
  const float c = 1.0f + ((float)j + 0.5f) * 0.015625f;  // exact
  const df64 u = (m - c) / (m + c);                   // |u| < 2^-8
  const df64 u2 = u * u;
  const float t = u2.hi;
  // log(m/c) = 2u + 2u^3 (1/3 + u^2/5 + u^4/7)
  const float tail = t * (0.2f + t * 0.14285714285714285f);
  const df64 P = df64{kDfThird_HI, kDfThird_LO} + tail;
  const df64 r = df_scale(u + u * u2 * P, 2.0f);
  const float2_ lc = kDfLogC[j];
  const df64 le = df64{kDfLn2_HI, kDfLn2_LO} * (float)e;
  return le + (df64{lc.x, lc.y} + r);
}

// Arctangent.
DF_HD df64 df_atan(df64 x) {
  const bool neg = x.hi < 0.0f;
  df64 z = neg ? -x : x;
  const bool inv = z.hi > 1.0f;
  if (inv) z = df_recip(z);
  int j = (int)(z.hi * 32.0f + 0.5f);
  j = j < 0 ? 0 : (j > 32 ? 32 : j);
  const float c = (float)j * 0.03125f;  // exact
  const df64 u = (z - c) / (df(1.0f) + z * c);  // |u| <= 1/64 (slightly more near the fold)
  const df64 u2 = u * u;
  const float t = u2.hi;
  // atan(u) = u + u^3 (-1/3 + u^2/5 - u^4/7 + u^6/9 - u^8/11)
  const float tail = t * (0.2f + t * (-0.14285714285714285f + t * (0.1111111111111111f - t * 0.09090909090909091f)));
  const df64 Q = df64{-kDfThird_HI, -kDfThird_LO} + tail;
  const df64 au = u + u * u2 * Q;
  const float2_ ac = kDfAtanC[j];
  df64 r = df64{ac.x, ac.y} + au;
  if (inv) r = df64{kDfPiHalf_HI, kDfPiHalf_LO} - r;
  return neg ? -r : r;
}

// ---------------------------------------------------------------------------
// Two df64 values at once, on GB300's packed FP32 instructions (add / mul / fma
// .f32x2: two lanes of a 64-bit register pair, each lane rounded as the scalar
// instruction does, so a lane holds the scalar form's bits).
//
// Why: a packed instruction takes the FMA pipe as long as two scalar ones but one
// issue slot and one 4-cycle latency (measured).  The pair kernels hold 8 warps
// per SM (255 registers), and their df64 code is chains of dependent additions:
// the FMA pipe was 46 % busy.
//
// DDD_F2_PLAIN: the same source on scalar instructions (tests compare the two).
#if defined(__CUDACC__) && !defined(DDD_F2_PLAIN)
struct f2 {
  unsigned long long v;
};
DF_HD f2 f2_make(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
DF_HD float f2_x(f2 a) { return __int_as_float((int)(unsigned)a.v); }
DF_HD float f2_y(f2 a) { return __int_as_float((int)(a.v >> 32)); }
DF_HD f2 operator+(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
DF_HD f2 operator-(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
DF_HD f2 operator*(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
DF_HD f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
DF_HD f2 operator-(f2 a) { return {a.v ^ 0x8000000080000000ull}; }
#else
struct f2 {
  float x, y;
};
DF_HD f2 f2_make(float x, float y) { return {x, y}; }
DF_HD float f2_x(f2 a) { return a.x; }
DF_HD float f2_y(f2 a) { return a.y; }
DF_HD f2 operator+(f2 a, f2 b) { return {a.x + b.x, a.y + b.y}; }
DF_HD f2 operator-(f2 a, f2 b) { return {a.x - b.x, a.y - b.y}; }
DF_HD f2 operator*(f2 a, f2 b) { return {a.x * b.x, a.y * b.y}; }
DF_HD f2 f2_fma(f2 a, f2 b, f2 c) { return {df_fma(a.x, b.x, c.x), df_fma(a.y, b.y, c.y)}; }
DF_HD f2 operator-(f2 a) { return {-a.x, -a.y}; }
#endif
DF_HD f2 f2_dup(float a) { return f2_make(a, a); }

struct df2 {
  f2 hi, lo;
};
DF_HD df2 df2_make(df64 x, df64 y) { return {f2_make(x.hi, y.hi), f2_make(x.lo, y.lo)}; }
DF_HD df2 df2_dup(df64 a) { return {f2_dup(a.hi), f2_dup(a.lo)}; }
DF_HD df64 df2_x(df2 a) { return {f2_x(a.hi), f2_x(a.lo)}; }
DF_HD df64 df2_y(df2 a) { return {f2_y(a.hi), f2_y(a.lo)}; }
DF_HD f2 f2_swap(f2 a) { return f2_make(f2_y(a), f2_x(a)); }
DF_HD df2 df2_swap(df2 a) { return {f2_swap(a.hi), f2_swap(a.lo)}; }

DF_HD df2 two_sum(f2 a, f2 b) {
  f2 s = a + b;
  f2 bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
DF_HD df2 two_diff(f2 a, f2 b) {  // two_sum(a, -b)
  f2 s = a - b;
  f2 bb = s - a;
  return {s, (a - (s - bb)) - (b + bb)};
}
DF_HD df2 fast_two_sum(f2 a, f2 b) {
  f2 s = a + b;
  return {s, b - (s - a)};
}
DF_HD df2 operator-(df2 a) { return {-a.hi, -a.lo}; }
DF_HD df2 operator+(df2 a, df2 b) {
  df2 s = two_sum(a.hi, b.hi);
  return fast_two_sum(s.hi, s.lo + (a.lo + b.lo));
}
DF_HD df2 operator-(df2 a, df2 b) {
  df2 s = two_diff(a.hi, b.hi);
  return fast_two_sum(s.hi, s.lo + (a.lo - b.lo));
}
DF_HD df2 operator+(df2 a, f2 b) {
  df2 s = two_sum(a.hi, b);
  return fast_two_sum(s.hi, s.lo + a.lo);
}
DF_HD df2 operator-(df2 a, f2 b) {
  df2 s = two_diff(a.hi, b);
  return fast_two_sum(s.hi, s.lo + a.lo);
}
DF_HD df2 operator*(df2 a, df2 b) {
  f2 p = a.hi * b.hi;
  f2 e = f2_fma(a.hi, b.hi, -p);
  e = f2_fma(a.hi, b.lo, e);
  e = f2_fma(a.lo, b.hi, e);
  return fast_two_sum(p, e);
}
DF_HD df2 operator*(df2 a, f2 b) {
  f2 p = a.hi * b;
  f2 e = f2_fma(a.hi, b, -p);
  e = f2_fma(a.lo, b, e);
  return fast_two_sum(p, e);
}
DF_HD df2 df_scale(df2 a, float p2) {
  const f2 s = f2_dup(p2);
  return {a.hi * s, a.lo * s};
}
DF_HD f2 df_qapprox(f2 a, f2 b) { return f2_make(df_qapprox(f2_x(a), f2_x(b)), df_qapprox(f2_y(a), f2_y(b))); }
DF_HD df2 operator/(df2 a, df2 b) {
  f2 q1 = df_qapprox(a.hi, b.hi);
  df2 r = a - b * q1;
  f2 q2 = df_qapprox(r.hi, b.hi);
  r = r - b * q2;
  f2 q3 = df_qapprox(r.hi, b.hi);
  return fast_two_sum(q1, q2) + q3;
}
DF_HD df2 df_recip(df2 b) { return df2{f2_dup(1.0f), f2_dup(0.0f)} / b; }

DF_HD df2 df_sqrt(df2 a) {
  const float ax = f2_x(a.hi), ay = f2_y(a.hi);
  if (!(ax > 0.0f && ay > 0.0f)) return df2_make(df_sqrt(df2_x(a)), df_sqrt(df2_y(a)));
  const f2 s = f2_make(df_sqrtf(ax), df_sqrtf(ay));
  const f2 p = s * s;
  const df2 r = a - df2{p, f2_fma(s, s, -p)};
  return fast_two_sum(s, df_qapprox(r.hi, f2_dup(2.0f) * s));
}

DF_HD df2 df_log(df2 a) {
  const int32_t bx = df_bits(f2_x(a.hi)), by = df_bits(f2_y(a.hi));
  const int32_t ex = ((bx >> 23) & 0xff) - 127, ey = ((by >> 23) & 0xff) - 127;
  const int32_t jx = (bx >> 17) & 63, jy = (by >> 17) & 63;
  const f2 scale = f2_make(df_from_bits((127 - ex) << 23), df_from_bits((127 - ey) << 23));
  const df2 m = {a.hi * scale, a.lo * scale};
  const f2 c = f2_dup(1.0f) + (f2_make((float)jx, (float)jy) + f2_dup(0.5f)) * f2_dup(0.015625f);
  const df2 u = (m - c) / (m + c);
  const df2 u2 = u * u;
  const f2 t = u2.hi;
  // Lane by lane: the compiler fuses a packed product that is used once into its sum,
  // also under --fmad=false.  Every other product here has two uses or more, or a power
  // of two as a factor (tests/test_df2_gpu.py compares all lanes on the device).
  auto poly = [](float w) { return w * (0.2f + w * 0.14285714285714285f); };
  const f2 tail = f2_make(poly(f2_x(t)), poly(f2_y(t)));
  const df2 P = df2{f2_dup(kDfThird_HI), f2_dup(kDfThird_LO)} + tail;
  const df2 r = df_scale(u + u * u2 * P, 2.0f);
  const float2_ lx = kDfLogC[jx], ly = kDfLogC[jy];
  const df2 le = df2{f2_dup(kDfLn2_HI), f2_dup(kDfLn2_LO)} * f2_make((float)ex, (float)ey);
  return le + (df2{f2_make(lx.x, ly.x), f2_make(lx.y, ly.y)} + r);
}

DF_HD df2 df_atan(df2 x) {
  const bool nx = f2_x(x.hi) < 0.0f, ny = f2_y(x.hi) < 0.0f;
  const f2 sg = f2_make(nx ? -1.0f : 1.0f, ny ? -1.0f : 1.0f);
  df2 z = {x.hi * sg, x.lo * sg};
  const bool ix = f2_x(z.hi) > 1.0f, iy = f2_y(z.hi) > 1.0f;
  if (ix || iy) {
    const df2 w = df_recip(z);
    z = {f2_make(ix ? f2_x(w.hi) : f2_x(z.hi), iy ? f2_y(w.hi) : f2_y(z.hi)),
         f2_make(ix ? f2_x(w.lo) : f2_x(z.lo), iy ? f2_y(w.lo) : f2_y(z.lo))};
  }
  int jx = (int)(f2_x(z.hi) * 32.0f + 0.5f), jy = (int)(f2_y(z.hi) * 32.0f + 0.5f);
  jx = jx < 0 ? 0 : (jx > 32 ? 32 : jx);
  jy = jy < 0 ? 0 : (jy > 32 ? 32 : jy);
  const f2 c = f2_make((float)jx, (float)jy) * f2_dup(0.03125f);
  const df2 one = {f2_dup(1.0f), f2_dup(0.0f)};
  const df2 u = (z - c) / (one + z * c);
  const df2 u2 = u * u;
  const f2 t = u2.hi;
  auto poly = [](float w) {
    return w * (0.2f + w * (-0.14285714285714285f + w * (0.1111111111111111f - w * 0.09090909090909091f)));
  };
  const f2 tail = f2_make(poly(f2_x(t)), poly(f2_y(t)));
  const df2 Q = df2{f2_dup(-kDfThird_HI), f2_dup(-kDfThird_LO)} + tail;
  const df2 au = u + u * u2 * Q;
  const float2_ cx = kDfAtanC[jx], cy = kDfAtanC[jy];
  df2 r = df2{f2_make(cx.x, cy.x), f2_make(cx.y, cy.y)} + au;
  const df2 w = df2{f2_dup(kDfPiHalf_HI), f2_dup(kDfPiHalf_LO)} - r;
  r = {f2_make(ix ? f2_x(w.hi) : f2_x(r.hi), iy ? f2_y(w.hi) : f2_y(r.hi)),
       f2_make(ix ? f2_x(w.lo) : f2_x(r.lo), iy ? f2_y(w.lo) : f2_y(r.lo))};
  return {r.hi * sg, r.lo * sg};
}

}  // namespace ddd
