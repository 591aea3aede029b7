// Seg-seg kernels whose unit of work is a step of 32 or 128 pairs, for calls that
// one CTA per 128 x 128 tile pair cannot spread over the GPU:
//   * the all-pairs force ("expanded": every pair's forces are stored and folded
//     afterwards) of small networks, and of larger ones the tile pairs beyond the
//     tile kernel's last full wave (not in the FMA build: ddd_internal.h),
//   * the index-list force (any size): one row segment against all others.
// Templated on the arithmetic policy of tile_body.cuh; the kernels have internal
// linkage because the strict and the FMA build compile this header with
// different flags.
//
// What bounds them: the tile kernel runs a tile pair's 128 steps one after the
// other in one CTA, 6.2 ms in strict FP64 whatever the network's size.  A
// 24-segment network is one tile pair, 512 segments are ten, so 151 and 142 of
// the 152 SMs idle.  One warp per 32 pairs gives 512 segments ~2,800 warps (8
// resident per SM at 255 registers), and 24 segments 23 warps of one step each.
#pragma once
#include <cstdint>

#include "tile_body.cuh"

namespace ddd {
namespace {

constexpr int XT = 128;               // tile of the all-pairs kernels
constexpr int XPOS = XT * XT;         // pair positions (step k, row t) of one tile pair
constexpr int kParCtas = 1216;        // near-parallel warps: 8 per SM
constexpr int64_t kQuadSegs = 64;     // four lanes per pair up to here

__device__ __forceinline__ void x_tile_index(int64_t b, int64_t& I, int64_t& J) {
  int64_t Jc = (int64_t)((sqrt(8.0 * (double)b + 1.0) - 1.0) * 0.5);
  while (Jc * (Jc + 1) / 2 > b) --Jc;
  while ((Jc + 1) * (Jc + 2) / 2 <= b) ++Jc;
  J = Jc;
  I = b - Jc * (Jc + 1) / 2;
}

// ---------------------------------------------------------------------------
// Expanded all-pairs.  Position (b, k, t) of tile pair b is the tile kernel's
// pair (row t, column (t + k) mod 128) of its step k; its forces are stored at
// vals[((b 128 + k) 12 + component) 128 + t] and its class in flags[(b 128 + k)
// 128 + t] (0 no pair, 1 general, 2 near-parallel).  x_fold adds them in the
// tile kernel's order, so both paths give the same bits.

// Class of every position by the reference's FP64 decision; the near-parallel
// positions also go into a list.  Its order does not matter: each entry is
// evaluated on its own and stored at its position.
__global__ void __launch_bounds__(256)
x_classify(const double* __restrict__ soa, const uint8_t* __restrict__ skip, int64_t npad, int64_t b0,
           uint8_t* __restrict__ flags, uint32_t* __restrict__ list, unsigned* __restrict__ count, unsigned long long* __restrict__ counters) {
  const uint32_t pos = blockIdx.x * 256u + threadIdx.x;
  const int t = pos & (XT - 1), k = (pos >> 7) & (XT - 1), jl = (t + k) & (XT - 1);
  int64_t I, J;
  x_tile_index(b0 + (pos >> 14), I, J);
  const int64_t i = I * XT + t, j = J * XT + jl;
  int f = 0;
  if (skip[i] == 0 && skip[j] == 0 && (I != J || jl > t)) {
    const D3 a = {soa[9 * npad + i], soa[10 * npad + i], soa[11 * npad + i]};
    const D3 b = {soa[9 * npad + j], soa[10 * npad + j], soa[11 * npad + j]};
    const double c = dot(a, b);
    f = 1.0 - c * c > kSqrtEps ? 1 : 2;
  }
  flags[pos] = (uint8_t)f;
  const unsigned par = __ballot_sync(0xffffffffu, f == 2), gen = __ballot_sync(0xffffffffu, f == 1);
  const int lane = threadIdx.x & 31;
  unsigned base = 0;
  if (lane == 0) {
    if (par) base = atomicAdd(count, (unsigned)__popc(par));
    if (counters) {
      if (gen) atomicAdd(&counters[0], (unsigned long long)__popc(gen));
      if (par) atomicAdd(&counters[1], (unsigned long long)__popc(par));
    }
  }
  base = __shfl_sync(0xffffffffu, base, 0);
  if (f == 2) list[base + __popc(par & ((1u << lane) - 1))] = pos;
}

// One warp per CTA.  The first kParCtas warps share the near-parallel list,
// every other one takes the 32 rows of a warp of one step: its general pairs.
// QUAD: 8 rows, four lanes per pair with a corner each.  A pair on its own is one
// chain of ~1,600 FP64 instructions at 64 cycles, 76 us; four lanes shorten it and
// repeat the rest of the pair's work, which pays while an SM has under two such
// warps: up to 64 segments (2,016 pairs).  24 segments: 150 -> 132 us per call; at
// 128 it costs 3 %.
template <class P, bool QUAD>
__global__ void __launch_bounds__(32)
x_pairs(TileArgs A, typename P::Consts KP, int64_t b0, const uint8_t* __restrict__ flags,
        const uint32_t* __restrict__ list, const unsigned* __restrict__ count, double* __restrict__ vals,
        unsigned long long* __restrict__ counters) {
  const int lane = threadIdx.x;
  if (blockIdx.x < kParCtas) {
    // Even CTAs take the forces on segment 1, odd ones those on segment 2: a short
    // list is bound by one side's chain of dependent operations, not by both.
    const unsigned n = *count, side = blockIdx.x & 1;
    unsigned long long nCore = 0;
    for (unsigned e = (blockIdx.x >> 1) * 32u + lane; e < n; e += kParCtas / 2 * 32u) {
      const uint32_t pos = list[e];
      const int t = pos & (XT - 1), k = (pos >> 7) & (XT - 1), jl = (t + k) & (XT - 1);
      int64_t I, J;
      x_tile_index(b0 + (pos >> 14), I, J);
      const SegF64 a = tb_load_seg64(A.soa, A.npad, I * XT + t), s = tb_load_seg64(A.soa, A.npad, J * XT + jl);
      D3 F1, F2;
      nCore += side ? parallel_pair_side<2>(A.K, a, s, F1, F2) : parallel_pair_side<1>(A.K, a, s, F1, F2);
      double* v = vals + ((int64_t)(pos >> 7) * 12 + 6 * side) * XT + t;
      v[0 * XT] = F1.x; v[1 * XT] = F1.y; v[2 * XT] = F1.z;
      v[3 * XT] = F2.x; v[4 * XT] = F2.y; v[5 * XT] = F2.z;
    }
    if (counters && nCore) atomicAdd(&counters[2], nCore);
    return;
  }
  const unsigned u = blockIdx.x - kParCtas;
  constexpr int kWarps = QUAD ? 16 : 4;  // per step
  const int64_t bk = u / kWarps;  // 128 b + k
  const int t = QUAD ? (int)(u % kWarps) * 8 + (lane >> 2) : (int)(u % kWarps) * 32 + lane;
  const bool act = flags[bk * XT + t] == 1;
  if (!__any_sync(0xffffffffu, act)) return;
  if (!QUAD && !act) return;  // a warp of quads stays whole: its lanes exchange corners
  int64_t I, J;
  x_tile_index(b0 + (bk >> 7), I, J);
  const int64_t i = I * XT + t, j = J * XT + ((t + (int)(bk & (XT - 1))) & (XT - 1));
  const typename P::Seg a = P::load_global(A, i), s = P::load_global(A, j);
  typename P::Scalar c;
  P::is_general(A, a, s, i, j, c);  // c; the class is the same FP64 decision
  typename P::Vec F1, F2, F3, F4;
  if constexpr (QUAD)
    P::template general<true, true>(KP, A, a, s, c, F1, F2, F3, F4);
  else
    P::template general<true>(KP, A, a, s, c, F1, F2, F3, F4);
  if (QUAD && (!act || (lane & 3))) return;
  double* v = vals + bk * 12 * XT + t;
  v[0 * XT] = P::pack(F1.x); v[1 * XT] = P::pack(F1.y); v[2 * XT] = P::pack(F1.z);
  v[3 * XT] = P::pack(F2.x); v[4 * XT] = P::pack(F2.y); v[5 * XT] = P::pack(F2.z);
  v[6 * XT] = P::pack(F3.x); v[7 * XT] = P::pack(F3.y); v[8 * XT] = P::pack(F3.z);
  v[9 * XT] = P::pack(F4.x); v[10 * XT] = P::pack(F4.y); v[11 * XT] = P::pack(F4.z);
}

// The slot of tile pair blockIdx.x / 12, component blockIdx.x % 12, from the
// stored pairs, in the tile kernel's order: a row segment's general pairs by
// step, then its near-parallel ones by step; a column segment's general pairs
// warp of rows by warp, by step within one, its near-parallel ones by row.  A
// thread takes 32 of its positions at a time: their classes as two masks, the values
// that hold a pair through asynchronous copies to shared memory, all in flight
// together (loaded to registers, the compiler takes each next to its use, one memory
// latency after another), then the sums, the near-parallel ones by set bit so that a
// warp issues no additions that no lane has.  One tile pair 20 -> 7 us, ten 55 -> 28.
// Only the first `live` rows and columns can hold pairs when there is one tile.
template <class P>
__global__ void __launch_bounds__(XT)
x_fold(const double* __restrict__ vals, const uint8_t* __restrict__ flags, int live, double* __restrict__ partial) {
  using Comp = typename P::Comp;
  __shared__ double buf[32][XT];  // each thread its own column
  const int64_t b = blockIdx.x / 12;
  const int c = blockIdx.x % 12, t = threadIdx.x;
  const bool row = c < 6;
  const double* v = vals + (b * XT * 12 + c) * XT;
  const uint8_t* f = flags + b * XPOS;
  const unsigned dst = (unsigned)__cvta_generic_to_shared(&buf[0][t]);
  Comp acc = P::comp_zero();
  double col = 0.0, fp = 0.0;
  for (int w = 0; 32 * w < live; ++w) {
    // Position u: step 32 w + u of row t, or row 32 w + u of column t.
    auto step = [&](int u) { return row ? 32 * w + u : (t - 32 * w - u) & (XT - 1); };
    auto lane = [&](int u) { return row ? t : 32 * w + u; };
    unsigned g = 0, p = 0;
#pragma unroll
    for (int u = 0; u < 32; ++u) {
      const unsigned k = f[step(u) * XT + lane(u)];
      g |= (k & 1) << u;
      p |= (k >> 1) << u;
    }
#pragma unroll
    for (int u = 0; u < 32; ++u)
      if ((g | p) >> u & 1)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + u * XT * 8),
                     "l"(v + (int64_t)step(u) * 12 * XT + lane(u))
                     : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
    // A column's rows of warp w in the order of the steps that pair them with it.
    const int first = row ? 0 : ((t >> 5) == w ? t & 31 : 31);
    if (!row) acc = P::comp_zero();
#pragma unroll
    for (int q = 0; q < 32; ++q) {
      const int u = row ? q : (first - q) & 31;
      if (g >> u & 1) acc = acc + P::unpack(buf[u][t]);
    }
    if (!row) col = w == 0 ? P::comp_to_double(acc) : col + P::comp_to_double(acc);
    for (; p; p &= p - 1) fp = fp + buf[__ffs(p) - 1][t];
    __syncwarp();  // the values are read before the next copies
  }
  partial[(b * 12 + c) * XT + t] = (row ? P::comp_to_double(acc) : col) + fp;
}

// Scratch of one expanded call: the pair values, the class bytes, the list and
// its length.
struct XScratch {
  double* vals;
  uint8_t* flags;
  uint32_t* list;
  unsigned* count;
  XScratch(void* p, int64_t nb) {
    char* q = (char*)p;
    vals = (double*)q;
    q += nb * XPOS * 12 * (int64_t)sizeof(double);
    list = (uint32_t*)q;
    q += nb * XPOS * (int64_t)sizeof(uint32_t);
    count = (unsigned*)q;
    q += 256;
    flags = (uint8_t*)q;
  }
};

// Classes, pairs and the slots (what the tile kernel writes) of tile pairs b0 to
// nb - 1, at most kExpandMaxPairs at a time through one scratch.
template <class P>
cudaError_t launch_expanded(const TileArgs& A, const typename P::Consts& KP, int64_t b0, int64_t nb, int64_t numSeg,
                            void* scratch, double* partial, unsigned long long* counters, cudaStream_t st) {
  const int live = nb == 1 ? (int)numSeg : XT;
  for (; b0 < nb; b0 += kExpandMaxPairs) {
    const int64_t n = nb - b0 < kExpandMaxPairs ? nb - b0 : kExpandMaxPairs;
    const XScratch x(scratch, n);
    cudaError_t e = cudaMemsetAsync(x.count, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    x_classify<<<(unsigned)(n * XPOS / 256), 256, 0, st>>>(A.soa, A.skip, A.npad, b0, x.flags, x.list, x.count,
                                                           counters);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if constexpr (P::kQuad) {
      if (numSeg <= kQuadSegs)
        x_pairs<P, true><<<kParCtas + XT * 16, 32, 0, st>>>(A, KP, b0, x.flags, x.list, x.count, x.vals, counters);
    }
    if (!P::kQuad || numSeg > kQuadSegs)
      x_pairs<P, false><<<(unsigned)(kParCtas + n * XT * 4), 32, 0, st>>>(A, KP, b0, x.flags, x.list, x.count, x.vals,
                                                                          counters);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    x_fold<P><<<(unsigned)(n * 12), XT, 0, st>>>(x.vals, x.flags, live, partial + b0 * 12 * XT);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Index rows (calcSegSegForce(..., idx), DislocationForces.jl:831-877): one CTA
// takes one row segment against m columns per thread, one column per thread and
// step, so no lane idles however few rows there are (the earlier tile form held one
// row per thread: 37 rows kept 37 of 128 lanes busy for 128 steps).
// Near-parallel columns are listed in shared memory (column order) and evaluated
// after the sweep: with ~5 % of the columns near-parallel, most CTAs have one
// warp's worth of them, where a list per warp would make every warp run both
// branches.  (37 rows x 6,001 segments: 570 us; one-warp CTAs of 128 columns, each
// with its list, 654.)  The threads' sums are added in a fixed tree; x_reduce_rows
// adds a row's blocks in a fixed order.
//
// df64 takes one CTA of 256 threads per SM when a call has many rows: its pair is
// ~10,000 instructions, several times what an SM holds, and two CTAs at different
// places of it fetched them twice (ncu: 1.3 instructions per cycle, half the warps'
// cycles without one).  The step's barriers keep the eight warps together.  6,001
// segments: 150 rows 0.838 -> 0.687 ms, 1,500 rows 7.18 -> 4.97, 6,001 rows 28.7 ->
// 19.5, where a row per thread had taken 2.5, 6.4 and 20.8.  The other forms lose 2 to
// 8 % so.
template <class P, int CT>
__global__ void __launch_bounds__(CT, 256 / CT)
x_rows(TileArgs A, typename P::Consts KP, const int64_t* __restrict__ rows, int64_t nBlk, int m,
       double* __restrict__ partial, unsigned long long* __restrict__ counters) {
  constexpr int NW = CT / 32;
  __shared__ uint16_t list[CT * kRowMaxSteps];
  __shared__ int cnt[NW];
  __shared__ double red[NW][6];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r = blockIdx.x / nBlk, j0 = (blockIdx.x % nBlk) * CT * m;
  const int64_t gi = rows[r];
  typename P::Acc f1 = P::acc_zero(), f2 = P::acc_zero();
  D3 p1 = {0, 0, 0}, p2 = {0, 0, 0};
  unsigned nGen = 0, nCore = 0;
  int nPar = 0;
  if (A.skip[gi] == 0) {
    const typename P::Seg a = P::load_global(A, gi);
    for (int q = 0; q < m; ++q) {
      const int64_t j = j0 + q * CT + tid;
      bool par = false;
      if (j < A.npad && A.skip[j] == 0 && j != gi) {
        const typename P::Seg s = P::load_global(A, j);
        typename P::Scalar c;
        if (P::is_general(A, a, s, gi, j, c)) {
          typename P::Vec F1, F2, F3, F4;
          P::template general<false>(KP, A, a, s, c, F1, F2, F3, F4);
          P::acc_add(f1, F1);
          P::acc_add(f2, F2);
          ++nGen;
        } else {
          par = true;
        }
      }
      const unsigned mask = __ballot_sync(0xffffffffu, par);
      if (lane == 0) cnt[warp] = __popc(mask);
      __syncthreads();
      int at = nPar;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        if (w < warp) at += cnt[w];
        nPar += cnt[w];
      }
      if (par) list[at + __popc(mask & ((1u << lane) - 1))] = (uint16_t)(q * CT + tid);
      __syncthreads();
    }
    if (tid < nPar) {
      const SegF64 b = tb_load_seg64(A.soa, A.npad, gi);
      for (int e = tid; e < nPar; e += CT) {
        const SegF64 s = tb_load_seg64(A.soa, A.npad, j0 + list[e]);
        D3 F1, F2;
        nCore += parallel_pair_side<1>(A.K, b, s, F1, F2);
        p1 = p1 + F1;
        p2 = p2 + F2;
      }
    }
  }
  const D3 g1 = P::acc_to_d3(f1) + p1, g2 = P::acc_to_d3(f2) + p2;
  double v[6] = {g1.x, g1.y, g1.z, g2.x, g2.y, g2.z};
  __syncwarp();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < 6; ++c) red[warp][c] = v[c];
  }
  __syncthreads();
  if (tid < 6) {
    double t = red[0][tid];
#pragma unroll
    for (int w = 1; w < NW; ++w) t += red[w][tid];
    partial[(int64_t)blockIdx.x * 6 + tid] = t;
  }
  if (counters) {
    nGen = __reduce_add_sync(0xffffffffu, nGen);
    nCore = __reduce_add_sync(0xffffffffu, nCore);
    if (lane == 0) {
      if (nGen) atomicAdd(&counters[0], (unsigned long long)nGen);
      if (nCore) atomicAdd(&counters[2], (unsigned long long)nCore);
      if (warp == 0 && nPar) atomicAdd(&counters[1], (unsigned long long)nPar);
    }
  }
}

// One warp per row: lane l adds blocks l, l + 32, ..., the lanes add in a tree.
__global__ void __launch_bounds__(128)
x_reduce_rows(const double* __restrict__ partial, int64_t nBlk, int64_t nRows, double* __restrict__ out) {
  const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= nRows) return;
  double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 2
  for (int64_t q = lane; q < nBlk; q += 32) {
    const double* p = partial + (r * nBlk + q) * 6;
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] += p[c];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < 6; ++c) out[6 * r + c] = v[c];
  }
}

template <class P>
cudaError_t launch_rows(const TileArgs& A, const typename P::Consts& KP, const int64_t* rows, int64_t nRows,
                        const RowPlan& plan, double* partial, double* out, unsigned long long* counters,
                        cudaStream_t st) {
  const unsigned grid = (unsigned)(nRows * plan.nBlk);
  if constexpr (P::kRowWide) {
    if (plan.threads == 256)
      x_rows<P, 256><<<grid, 256, 0, st>>>(A, KP, rows, plan.nBlk, plan.m, partial, counters);
  }
  if (plan.threads == 128) x_rows<P, 128><<<grid, 128, 0, st>>>(A, KP, rows, plan.nBlk, plan.m, partial, counters);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  x_reduce_rows<<<(unsigned)((nRows + 3) / 4), 128, 0, st>>>(partial, plan.nBlk, nRows, out);
  return cudaGetLastError();
}

}  // namespace
}  // namespace ddd
