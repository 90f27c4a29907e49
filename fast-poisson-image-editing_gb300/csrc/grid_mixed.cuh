// The last fold of a mixed-precision step and the residual norms (grid_mixed.cu).
#pragma once

#include "common.cuh"
#include "grid_kernels.cuh"

namespace fpie {

// xout = xin + e where a group of 4 pixels has masked ones; e in FP16 or BF16
// by the precision.
void launch_fold(int precision, const GridLaunch& L, const GridGeom& G, const uint8_t* mask,
                 const float* xin, const void* e, float* xout, cudaStream_t st);

// out[0..2] = max |residual| of x per channel, out[3..5] = sum |residual|
// (device or pinned memory).  parts: 6 * L.nparts doubles of scratch; count: a
// device word that is 0 between launches; flag, unless NULL, goes to out[6].
void launch_norms(const GridLaunch& L, const GridGeom& G, const uint8_t* mask, const float* g,
                  const float* x, double* parts, unsigned* count, double* out, cudaStream_t st,
                  const int* flag = nullptr);

}  // namespace fpie
