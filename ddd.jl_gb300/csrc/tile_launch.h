// Host entries of the tile body's persistent kernels (tile_launch.cu): the exact
// passes of the surrogate path and the batched tiles, for the FP64 policies (their
// near pass apart) and the df64 ones.
#pragma once
#include "tile_body.cuh"

namespace ddd {

// pol: 0 or 1 of the group (strict, fast; df64, f32c).
#define DDD_NEAR_DECLS \
  /* The near pass: tile_body's MODE 2. */ \
  cudaError_t near_launch(int pol, const TileArgs& A, const int4* items, const int32_t* nDev, int32_t nHost, \
                          int32_t* next, double* partial, unsigned long long* counters, int grid, cudaStream_t st); \
  /* Its resident CTAs per SM; loads it. */ \
  cudaError_t near_occupancy(int* per);
#define DDD_TILE_DECLS \
  cudaError_t exact_launch(int pol, const TileArgs& A, const int4* items, const int32_t* nDev, int32_t nHost, \
                           int32_t* next, double* partial, unsigned long long* counters, int grid, cudaStream_t st); \
  /* T = 64 or 128; *grid = persistent CTAs for nItems; outside any capture. */ \
  cudaError_t batch_prepare(int pol, int T, int device, int64_t nItems, unsigned* grid); \
  cudaError_t batch_launch(int pol, int T, const TileArgs& A, unsigned grid, const int4* items, int32_t nItems, \
                           int32_t* next, double* partial, unsigned long long* counters, cudaStream_t st);

namespace near_tiles {
DDD_NEAR_DECLS
}
namespace f64_tiles {
DDD_TILE_DECLS
}
namespace df_tiles {
DDD_NEAR_DECLS
DDD_TILE_DECLS
}
#undef DDD_NEAR_DECLS
#undef DDD_TILE_DECLS

}  // namespace ddd
