// Launch plans for the grid sweep / finish kernels (grid_kernels.cu).
#pragma once

#include "common.cuh"

namespace fpie {

struct GridLaunch {
  dim3 sweep_block, sweep_grid;    // one-sweep kernel
  dim3 finish_block, finish_grid;  // residual + image kernel
  int finish_rows;                 // rows per thread of the latter
  int nparts;                      // residual partials: sweep_grid's blocks, finish_grid has no more
};

GridLaunch grid_launch(const GridGeom& G);

// One Jacobi sweep xin -> xout over the crop (all three channels).
void launch_grid_sweep(const GridLaunch& L, const GridGeom& G,
                       const uint8_t* mask, const float* g, const float* xin,
                       float* xout, cudaStream_t st);

// The residual sums (err[3]; parts: nparts x 3 doubles of scratch, count: a
// device word that is 0 between launches) and the clipped uint8 image in the
// reference's interleaved [n][m][3] layout.  err may be pinned host memory;
// flag, unless NULL, is copied to err[3].
void launch_grid_finish(const GridLaunch& L, const GridGeom& G,
                        const uint8_t* mask, const float* g, const float* x,
                        uint8_t* img, double* parts, unsigned* count, float* err,
                        cudaStream_t st, const int* flag = nullptr);

}  // namespace fpie
