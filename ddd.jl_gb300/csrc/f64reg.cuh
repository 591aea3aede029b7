// rd: a double whose additions, subtractions and products are issued as
// three-register FP64 FMAs, with the bits of the plain operations:
//   a + b = fma(a, 1, b),   a - b = fma(b, -1, a),   a b = fma(a, b, -0).
// (The product is exact inside the FMA, so each rounds once, as the plain
// operation does; -0 keeps the sign of a zero product.)
//
// Why: measured on one GB300 with 8 resident warps per SM, an FP64 FMA whose
// three operands are registers takes 16.0 cycles of an SM's FP64 pipe per warp;
// DADD, DMUL and an FMA with an immediate or constant-bank operand take 19.0.
// The pair kernels are bound by that pipe and mostly add and multiply.
//
// Measured with it (16,384 segments; 4,096 segments x 65,536 points), same bits:
// strict pairs 3.12e8 -> 3.39e8/s, fast 5.45e8 -> 5.76e8, strict stress
// 1.67e9 -> 1.87e9 evaluations/s, fast 3.98e9 -> 4.6e9.
//
// 1 and -0 must be per-thread registers: a uniform register costs the 19 cycles
// too, and the compiler moves a value that it knows to be the same in every lane
// there (a constant, a load from one address).  So each lane loads its own copy.
//
// Translation units that want the compiler's own operators (to be contracted in the
// FMA build, or for the registers: build.py) define DDD_F64_PLAIN; a host compiler
// gets plain double.
#pragma once
#include <cstdint>

namespace ddd {

#if defined(__CUDACC__) && !defined(DDD_F64_PLAIN)

#define DDD_X8(v) v, v, v, v, v, v, v, v
static __device__ double kF64Ones[32] = {DDD_X8(1.0), DDD_X8(1.0), DDD_X8(1.0), DDD_X8(1.0)};
static __device__ double kF64NegZeros[32] = {DDD_X8(-0.0), DDD_X8(-0.0), DDD_X8(-0.0), DDD_X8(-0.0)};
#undef DDD_X8

struct rd {
  double v;
  rd() = default;
  __device__ __forceinline__ rd(double a) : v(a) {}
  __device__ __forceinline__ operator double() const { return v; }
};
__device__ __forceinline__ rd rd_one() { return __ldg(&kF64Ones[threadIdx.x & 31]); }
__device__ __forceinline__ double rd_nzero() { return __ldg(&kF64NegZeros[threadIdx.x & 31]); }

__device__ __forceinline__ rd operator+(rd a, rd b) { return __fma_rn(a.v, rd_one().v, b.v); }
__device__ __forceinline__ rd operator-(rd a, rd b) { return __fma_rn(-b.v, rd_one().v, a.v); }
__device__ __forceinline__ rd operator*(rd a, rd b) { return __fma_rn(a.v, b.v, rd_nzero()); }
__device__ __forceinline__ rd operator/(rd a, rd b) { return a.v / b.v; }
__device__ __forceinline__ rd operator-(rd a) { return -a.v; }
__device__ __forceinline__ rd operator+(double a, rd b) { return rd(a) + b; }
__device__ __forceinline__ rd operator+(rd a, double b) { return a + rd(b); }
__device__ __forceinline__ rd operator-(double a, rd b) { return rd(a) - b; }
__device__ __forceinline__ rd operator-(rd a, double b) { return a - rd(b); }
__device__ __forceinline__ rd operator*(double a, rd b) { return rd(a) * b; }
__device__ __forceinline__ rd operator*(rd a, double b) { return a * rd(b); }
__device__ __forceinline__ rd operator/(double a, rd b) { return a / b.v; }
__device__ __forceinline__ rd operator/(rd a, double b) { return a.v / b; }
__device__ __forceinline__ rd& operator+=(rd& a, rd b) { return a = a + b; }
__device__ __forceinline__ rd sqrt(rd a) { return ::sqrt(a.v); }
__device__ __forceinline__ rd twice(rd a) { return a + a; }

#elif defined(__CUDACC__)

typedef double rd;
__device__ __forceinline__ rd rd_one() { return 1.0; }
__device__ __forceinline__ rd twice(rd a) { return 2.0 * a; }

#else

typedef double rd;
inline rd rd_one() { return 1.0; }
inline rd twice(rd a) { return 2.0 * a; }

#endif

}  // namespace ddd
