// Refinement kernels of the mixed-precision grid form (grid_mixed.cu).
#pragma once

#include "common.cuh"
#include "grid_kernels.cuh"

namespace fpie {

// x_out = x_in + e (masked pixels; e may be NULL for no fold), r = FP32
// residual of the folded state (r may be NULL).  Launch geometry: the one-sweep
// kernel's (grid_launch(G).sweep_grid / sweep_block).
void launch_refine(int precision, dim3 grid, dim3 block, const GridGeom& G, const uint8_t* mask,
                   const float* g, const float* xin, const void* e, float* xout, float* r,
                   cudaStream_t st);

// out[0..2] = max |residual| of x per channel, out[3..5] = sum |residual|
// (device or pinned memory).  parts: 6 * L.nparts doubles of scratch; count: a
// device word that is 0 between launches; flag, unless NULL, goes to out[6].
void launch_norms(const GridLaunch& L, const GridGeom& G, const uint8_t* mask, const float* g,
                  const float* x, double* parts, unsigned* count, double* out, cudaStream_t st,
                  const int* flag = nullptr);

}  // namespace fpie
