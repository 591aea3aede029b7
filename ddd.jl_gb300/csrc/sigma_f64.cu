// FP64 field-point stress σ̃ (calc_σTilde, DislocationFEM.jl:86-303).
//
// One thread per field point; segments stream through shared memory in tiles
// of SIG_TILE, every thread reading the same segment at the same time (a
// broadcast).  Each point's six components accumulate in registers over the
// segments in list order — the same per-point summation order as the
// reference's segment-outer loop — and are written once (48 B/point), so σ
// never round-trips through memory per segment as it does on the CPU.  Calls with
// too few points for that take sigma_split.
#include <cuda_runtime.h>

#include <atomic>

#include "ddd_internal.h"
#include "pair_f64.cuh"

// Compiled twice, like segseg_f64.cu: strict (--fmad=false) and fast (FMA).
#ifndef DDD_VARIANT
#define DDD_VARIANT strict
#endif

namespace ddd {
namespace DDD_VARIANT {

// One warp per CTA: each thread owns a point and the CTA's 32 points share a
// 32-segment tile in shared memory.  Small CTAs spread a small point set evenly
// over the SMs (32,768 points: 1,024 CTAs, 6.7 per SM, where 128-thread CTAs
// left 48 SMs with one CTA and 104 with two); each point still adds the
// segments in order 0..nSeg-1.  24 resident CTAs per SM cap registers at 85,
// the budget the 128-thread form ran at (80).
constexpr int SIG_TILE = 32;

__global__ void __launch_bounds__(SIG_TILE, 24)
sigma_tilde_f64(KConsts K, const double* __restrict__ soa, int64_t npad, int64_t nSeg, const double* __restrict__ x0,
                int64_t M, double* __restrict__ sigma) {
  __shared__ double seg[15][SIG_TILE];  // n1, n2, b, t, t x b
  const int t = threadIdx.x;
  const int64_t j = blockIdx.x * (int64_t)SIG_TILE + t;
  D3 x = {0, 0, 0};
  if (j < M) x = {x0[3 * j], x0[3 * j + 1], x0[3 * j + 2]};
  rd sig[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int64_t s0 = 0; s0 < nSeg; s0 += SIG_TILE) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 12; ++k) seg[k][t] = soa[k * npad + s0 + t];
    {
      const D3 tx = cross(D3{seg[9][t], seg[10][t], seg[11][t]}, D3{seg[6][t], seg[7][t], seg[8][t]});
      seg[12][t] = tx.x;
      seg[13][t] = tx.y;
      seg[14][t] = tx.z;
    }
    __syncthreads();
    const int n = (int)min((int64_t)SIG_TILE, nSeg - s0);
    if (j < M) {
      for (int q = 0; q < n; ++q) {
        D3 n1 = {seg[0][q], seg[1][q], seg[2][q]};
        D3 n2 = {seg[3][q], seg[4][q], seg[5][q]};
        D3 b = {seg[6][q], seg[7][q], seg[8][q]};
        D3 tt = {seg[9][q], seg[10][q], seg[11][q]};
        D3 txb = {seg[12][q], seg[13][q], seg[14][q]};
        sigma_point(K, b, n1, n2, tt, txb, x, sig);
      }
    }
  }
  if (j < M) {
#pragma unroll
    for (int c = 0; c < 6; ++c) sigma[6 * j + c] = sig[c];
  }
}

// Fewer points than kSigmaSplitPoints: a thread per (segment, point) instead of
// per point, segments in chunks of `chunk` evaluations (sigma_split_chunk).  The
// contributions go to a store and are added to sigma in segment order by the first
// blocks of the next chunk's launch, beside its evaluations (one DADD of a point's
// chain takes 64 cycles, so a chunk's chain is ~1/10 of its evaluations' time), so
// every point's sum keeps the reference's order, and in the strict build its bits
// (the FMA build contracts an evaluation differently in the two kernels: 4e-16 of
// the largest stress).  Two stores alternate.
//
// Why: a point per thread is 20 one-warp CTAs for 613 points, one warp per SM at
// 64 cycles per FP64 instruction (its latency) instead of 16-19 (the pipe's
// rate); four warps per SM saturate the pipe.  613 points x 4,096 segments took
// 38.5 ms and takes 1.3; 24,000 points x 8,192 segments 124 (3.9 warps per SM, 5
// on some) and 101.  At 32,768 points both forms run at 1.93e9-1.95e9/s.
__global__ void __launch_bounds__(SIG_TILE, 24)
sigma_split(KConsts K, const double* __restrict__ soa, int64_t npad, const double* __restrict__ txb,
            const double* __restrict__ x0, unsigned M, unsigned addBlocks, const double* __restrict__ prev,
            unsigned prevSegs, bool first, double* __restrict__ sigma, double* __restrict__ store, int64_t chunk,
            int64_t s0, unsigned segs) {
  if (blockIdx.x < addBlocks) {
    const unsigned q = blockIdx.x * SIG_TILE + threadIdx.x;
    if (q >= 6 * M) return;
    const unsigned c = q / M, j = q % M;
    const double* p = prev + c * chunk + j;
    double acc = first ? 0.0 : sigma[6 * (int64_t)j + c];
#pragma unroll 16
    for (unsigned s = 0; s < prevSegs; ++s) acc += p[s * M];
    sigma[6 * (int64_t)j + c] = acc;
    return;
  }
  const unsigned e = (blockIdx.x - addBlocks) * SIG_TILE + threadIdx.x;
  if (e >= segs * M) return;
  const unsigned s = e / M, j = e % M;
  const double* g = soa + s0 + s;
  const double* x = x0 + 3 * (int64_t)j;
  rd sig[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const double* tx = txb + s0 + s;
  sigma_point(K, D3{g[6 * npad], g[7 * npad], g[8 * npad]}, D3{g[0], g[npad], g[2 * npad]},
              D3{g[3 * npad], g[4 * npad], g[5 * npad]}, D3{g[9 * npad], g[10 * npad], g[11 * npad]},
              D3{tx[0], tx[npad], tx[2 * npad]}, D3{x[0], x[1], x[2]}, sig);
#pragma unroll
  for (int c = 0; c < 6; ++c) store[c * chunk + e] = sig[c];
}

// t x b of every segment (3 x npad), as the point kernel forms it per tile.
__global__ void sigma_txb(const double* __restrict__ soa, int64_t npad, double* __restrict__ txb) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= npad) return;
  const D3 v = cross(D3{soa[9 * npad + i], soa[10 * npad + i], soa[11 * npad + i]},
                     D3{soa[6 * npad + i], soa[7 * npad + i], soa[8 * npad + i]});
  txb[i] = v.x;
  txb[npad + i] = v.y;
  txb[2 * npad + i] = v.z;
}

cudaError_t launch_sigma_f64(const KConsts& K, const double* soa, int64_t npad, int64_t nSeg, const double* x0,
                             int64_t M, double* sigma, int64_t chunk, double* scratch, cudaStream_t st) {
  if (M == 0) return cudaSuccess;
  if (!scratch) {
    sigma_tilde_f64<<<(unsigned)((M + SIG_TILE - 1) / SIG_TILE), SIG_TILE, 0, st>>>(K, soa, npad, nSeg, x0, M, sigma);
    return cudaGetLastError();
  }
  // Loaded here too: a later call under stream capture has no scratch.
  static std::atomic<uint64_t> loaded{0};
  const cudaError_t le = set_smem_once(sigma_tilde_f64, 0, loaded);
  if (le != cudaSuccess) return le;
  double* store[2] = {scratch, scratch + 6 * chunk};
  double* txb = scratch + 12 * chunk;
  sigma_txb<<<(unsigned)((npad + 255) / 256), 256, 0, st>>>(soa, npad, txb);
  const int64_t step = chunk / M;
  const unsigned addBlocks = (unsigned)((6 * M + SIG_TILE - 1) / SIG_TILE);
  unsigned prevSegs = 0;
  int turn = 0;
  for (int64_t s0 = 0; s0 < nSeg || prevSegs; s0 += step, ++turn) {
    const unsigned segs = s0 < nSeg ? (unsigned)(nSeg - s0 < step ? nSeg - s0 : step) : 0;
    const unsigned add = prevSegs ? addBlocks : 0;
    const unsigned eval = (unsigned)((segs * M + SIG_TILE - 1) / SIG_TILE);
    sigma_split<<<add + eval, SIG_TILE, 0, st>>>(K, soa, npad, txb, x0, (unsigned)M, add, store[(turn + 1) & 1],
                                                 prevSegs, turn == 1, sigma, store[turn & 1], chunk, s0, segs);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    prevSegs = segs;
  }
  return cudaSuccess;
}

}  // namespace DDD_VARIANT
}  // namespace ddd
