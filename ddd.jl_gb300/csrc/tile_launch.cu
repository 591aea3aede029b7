// Persistent kernels over tile pairs: CTAs take work items from a global counter
// (one atomicAdd per item, no waiting) and run the shared tile body on each.
// Compiled three times, with --fmad=false: the FP64 policies with f64reg.cuh's
// operators; the df64 ones (DDD_DF_POLICIES) with plain ones, whose two constants
// their FP32 main loop has no registers for; and the near pass of the FP64 ones
// (DDD_NEAR_PASS) with plain ones too: its dense chunks hold few pairs, and a
// pair that starts with those constants' loads and spills took the whole call of
// 32,768 segments with the 2-point far field from 53.2 to 59.3 ms (fast FP64 near
// pairs; 75.0 to 78.2 strict).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "ddd_internal.h"
#include "tile_launch.h"
#ifdef DDD_DF_POLICIES
#include "tile_pol_df.cuh"
#define DDD_TILE_NS df_tiles
#elif defined(DDD_NEAR_PASS)
#include "tile_pol_fx.cuh"
#define DDD_TILE_NS near_tiles
#else
#include "tile_pol_fx.cuh"
#define DDD_TILE_NS f64_tiles
#endif

namespace ddd {
namespace DDD_TILE_NS {

#ifdef DDD_DF_POLICIES
using Pol0 = PolDF<0>;
using Pol1 = PolDF<1>;
template <class P>
typename P::Consts consts(const KConsts& K) {
  return {kconsts_df(K), kconsts_f(K)};
}
#else
using Pol0 = PolF64;
using Pol1 = PolF64Fast;
template <class P>
typename P::Consts consts(const KConsts&) {
  return {};
}
#endif

// Work item: (slot, first row segment, first column segment, diagonal flag); the
// item count is read from the device (nDev) when given.
template <int T, int MODE, class P>
__global__ void __launch_bounds__(T, 256 / T)
persistent_tiles(TileArgs A, typename P::Consts KP, const int4* __restrict__ items, const int32_t* __restrict__ nDev,
                 int32_t nHost, int32_t* __restrict__ next, double* __restrict__ partial,
                 unsigned long long* __restrict__ counters) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<TileSmemT<T, P>*>(smem_raw);
  __shared__ int32_t s_item;
  const int32_t nItems = nDev ? *nDev : nHost;
  for (;;) {
    __syncthreads();  // the previous item's shared memory is no longer read
    if (threadIdx.x == 0) s_item = atomicAdd(next, 1);
    __syncthreads();
    const int32_t w = s_item;
    if (w >= nItems) break;
    const int4 it = items[w];
    tile_body<T, MODE, P>(A, KP, sm, it.y, it.z, it.w != 0, partial + (int64_t)it.x * 12 * T, counters);
  }
}

template <int T, int MODE, class P>
static cudaError_t set_attr() {
  static std::atomic<uint64_t> done{0};
  return set_smem_once(persistent_tiles<T, MODE, P>, (int)sizeof(TileSmemT<T, P>), done);
}

template <int T, int MODE, class P>
static cudaError_t launch(const TileArgs& A, const int4* items, const int32_t* nDev, int32_t nHost, int32_t* next,
                          double* partial, unsigned long long* counters, unsigned grid, cudaStream_t st) {
  const cudaError_t e = set_attr<T, MODE, P>();
  if (e != cudaSuccess) return e;
  persistent_tiles<T, MODE, P><<<grid, T, sizeof(TileSmemT<T, P>), st>>>(A, consts<P>(A.K), items, nDev, nHost, next,
                                                                         partial, counters);
  return cudaGetLastError();
}

#if defined(DDD_NEAR_PASS) || defined(DDD_DF_POLICIES)
cudaError_t near_launch(int pol, const TileArgs& A, const int4* items, const int32_t* nDev, int32_t nHost,
                        int32_t* next, double* partial, unsigned long long* counters, int grid, cudaStream_t st) {
  return pol ? launch<128, 2, Pol1>(A, items, nDev, nHost, next, partial, counters, grid, st)
             : launch<128, 2, Pol0>(A, items, nDev, nHost, next, partial, counters, grid, st);
}

cudaError_t near_occupancy(int* per) {
  const cudaError_t e = set_attr<128, 2, Pol0>();
  return e != cudaSuccess ? e
                          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, persistent_tiles<128, 2, Pol0>, 128,
                                                                          sizeof(TileSmemT<128, Pol0>));
}
#endif

#ifndef DDD_NEAR_PASS
template <int T, class P>
static cudaError_t prepare(int device, int64_t nItems, unsigned* grid) {
  cudaError_t e = set_attr<T, 0, P>();
  int sms = 0, per = 0;
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, persistent_tiles<T, 0, P>, T, sizeof(TileSmemT<T, P>));
  if (e != cudaSuccess) return e;
  const int64_t want = (int64_t)sms * std::max(per, 1);
  *grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, nItems));
  return cudaSuccess;
}

cudaError_t exact_launch(int pol, const TileArgs& A, const int4* items, const int32_t* nDev, int32_t nHost,
                         int32_t* next, double* partial, unsigned long long* counters, int grid, cudaStream_t st) {
  return pol ? launch<128, 0, Pol1>(A, items, nDev, nHost, next, partial, counters, grid, st)
             : launch<128, 0, Pol0>(A, items, nDev, nHost, next, partial, counters, grid, st);
}

cudaError_t batch_prepare(int pol, int T, int device, int64_t nItems, unsigned* grid) {
  if (T == 64) return pol ? prepare<64, Pol1>(device, nItems, grid) : prepare<64, Pol0>(device, nItems, grid);
  return pol ? prepare<128, Pol1>(device, nItems, grid) : prepare<128, Pol0>(device, nItems, grid);
}

cudaError_t batch_launch(int pol, int T, const TileArgs& A, unsigned grid, const int4* items, int32_t nItems,
                         int32_t* next, double* partial, unsigned long long* counters, cudaStream_t st) {
  if (T == 64)
    return pol ? launch<64, 0, Pol1>(A, items, nullptr, nItems, next, partial, counters, grid, st)
               : launch<64, 0, Pol0>(A, items, nullptr, nItems, next, partial, counters, grid, st);
  return pol ? launch<128, 0, Pol1>(A, items, nullptr, nItems, next, partial, counters, grid, st)
             : launch<128, 0, Pol0>(A, items, nullptr, nItems, next, partial, counters, grid, st);
}
#endif

}  // namespace DDD_TILE_NS
}  // namespace ddd
