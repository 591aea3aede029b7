// Host entries of the tile body's persistent kernels (tile_launch.cu): the exact
// passes of the surrogate path and the batched tiles, for the FP64 policies and,
// compiled apart, for the df64 ones.
#pragma once
#include "tile_body.cuh"

namespace ddd {

#define DDD_TILE_DECLS \
  /* pol: 0 or 1 of the group (strict, fast; df64, f32c); mode: tile_body's MODE, 0 or 2. */ \
  cudaError_t exact_launch(int pol, int mode, const TileArgs& A, const int4* items, const int32_t* nDev, \
                           int32_t nHost, int32_t* next, double* partial, unsigned long long* counters, int grid, \
                           cudaStream_t st); \
  /* Resident CTAs per SM of the near pass; loads it. */ \
  cudaError_t exact_occupancy(int* per); \
  /* T = 64 or 128; *grid = persistent CTAs for nItems; outside any capture. */ \
  cudaError_t batch_prepare(int pol, int T, int device, int64_t nItems, unsigned* grid); \
  cudaError_t batch_launch(int pol, int T, const TileArgs& A, unsigned grid, const int4* items, int32_t nItems, \
                           int32_t* next, double* partial, unsigned long long* counters, cudaStream_t st);

namespace f64_tiles {
DDD_TILE_DECLS
}
namespace df_tiles {
DDD_TILE_DECLS
}
#undef DDD_TILE_DECLS

}  // namespace ddd
