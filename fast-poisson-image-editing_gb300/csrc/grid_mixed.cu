// Mixed-precision iterative refinement for the grid form.
//
// The FP32 solution x is kept; every cycle
//   1. refine: x <- x + e (e: the correction, FP16 or BF16), then the FP32
//      residual r = grad + up + down + left + right - 4x on masked pixels (in
//      the cycle's first inner launch, grid_tbp.cu);
//   2. inner: Jacobi sweeps on the correction equation 4e - sum(e_nb) = r,
//      e starting at 0 and kept at 0 on unmasked pixels, FP32 arithmetic,
//      e stored in FP16/BF16 between launches (grid_tbp.cu, storage type TS).
// Here: the fold that ends a step, and the norms that decide convergence (max
// |r| and sum |r| per channel, with at least a double's bits).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "grid_mixed.cuh"

namespace fpie {

template <typename TS>
__device__ __forceinline__ float to_f(TS v);
template <>
__device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename TS>
__device__ __forceinline__ float4 ld4_any(const TS* p) {
  return make_float4(to_f(p[0]), to_f(p[1]), to_f(p[2]), to_f(p[3]));
}

// The fold that ends a step: xout = xin + e.  Thread = 4 adjacent pixels of one
// row, all channels (the one-sweep kernel's geometry).
template <typename TS>
__global__ void __launch_bounds__(256)
grid_fold_kernel(GridGeom G, const uint8_t* __restrict__ mask, const float* __restrict__ xin,
                 const TS* __restrict__ e, float* __restrict__ xout) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= G.n || 4 * q >= G.m) return;
  const long long p = G.at(i, 4 * q);
  if (*reinterpret_cast<const uint32_t*>(mask + p) == 0) return;  // unmasked pixels have e = 0
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const long long o = c * G.plane + p;
    const float4 x = ld4(xin + o), d = ld4_any(e + o);
    *reinterpret_cast<float4*>(xout + o) = make_float4(__fadd_rn(x.x, d.x), __fadd_rn(x.y, d.y),
                                                       __fadd_rn(x.z, d.z), __fadd_rn(x.w, d.w));
  }
}

// ---- residual norms ------------------------------------------------------------
// max |r| and sum |r| per channel of the state x, out[0..2] and out[3..5]; the
// last block to arrive reduces the blocks' partials (6 doubles each) in a fixed
// order.  One launch: with a second one for the blocks and FP64 reductions a
// check of a 152x152 grid took 14 us.
__global__ void __launch_bounds__(256)
grid_norms_kernel(GridGeom G, const uint8_t* __restrict__ mask, const float* __restrict__ g,
                  const float* __restrict__ x, double* __restrict__ parts,
                  unsigned* __restrict__ count, double* __restrict__ out, const int* flag,
                  int rows) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int i0 = (blockIdx.y * blockDim.y + threadIdx.y) * rows;
  const int i1 = 4 * q < G.m ? min(i0 + rows, G.n) : i0;
  float mx[3] = {0.f, 0.f, 0.f};
  Sum3 sm[3];
  // Values above 2^90, whose float sum could overflow where a double's does not.
  double huge[3] = {0.0, 0.0, 0.0};
  for (int i = i0; i < i1; ++i) {
    const long long p = G.at(i, 4 * q);
    const uint32_t mk = __ldg(reinterpret_cast<const uint32_t*>(mask + p));
    if (!mk) continue;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float* xc = x + c * G.plane + p;
      const float4 ce = ld4(xc), up = ld4(xc - G.pitch), dn = ld4(xc + G.pitch);
      const float4 gg = ld4(g + c * G.plane + p);
      const float xv[6] = {__ldg(xc - 1), ce.x, ce.y, ce.z, ce.w, __ldg(xc + 4)};
      const float uv[4] = {up.x, up.y, up.z, up.w}, dv[4] = {dn.x, dn.y, dn.z, dn.w};
      const float gv[4] = {gg.x, gg.y, gg.z, gg.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if ((mk >> (8 * k)) & 0xffu) {
          const float v = fabsf(grid_res(xv[k + 1], gv[k], uv[k], dv[k], xv[k], xv[k + 2]));
          mx[c] = fmaxf(mx[c], v);
          if (v > 0x1p90f)
            huge[c] += (double)v;
          else
            sum3_add(sm[c], v);
        }
    }
  }
  __shared__ float shm[3][8];
  __shared__ double shs[3][8];
  __shared__ bool last;
  const int tid = threadIdx.x + threadIdx.y * blockDim.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    // Not negative and no NaN (a maximum drops them): bits order as values do.
    const float m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx[c])));
    const bool any = __any_sync(0xffffffffu, huge[c] != 0.0);
    sum3_warp(sm[c]);
    if (any)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) huge[c] += __shfl_down_sync(0xffffffffu, huge[c], o);
    if (lane == 0) {
      shm[c][warp] = m;
      shs[c][warp] = sum3_value(sm[c]) + huge[c];
    }
  }
  __syncthreads();
  const unsigned block = blockIdx.y * gridDim.x + blockIdx.x, blocks = gridDim.x * gridDim.y;
  if (tid < 3) {
    float m = 0.f;
    double t = 0.0;
    for (int w = 0; w < 8; ++w) {
      m = fmaxf(m, shm[tid][w]);
      t += shs[tid][w];
    }
    parts[6 * (size_t)block + tid] = (double)m;
    parts[6 * (size_t)block + 3 + tid] = t;
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last = atomicAdd(count, 1u) == blocks - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // A warp per column of the partials: lanes stride over the blocks.
  if (warp < 6) {
    double v = 0.0;
    for (unsigned k = lane; k < blocks; k += 32) {
      const double u = __ldcg(parts + 6 * (size_t)k + warp);
      v = warp < 3 ? fmax(v, u) : v + u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double u = __shfl_down_sync(0xffffffffu, v, o);
      v = warp < 3 ? fmax(v, u) : v + u;
    }
    if (lane == 0) out[warp] = v;
  }
  // Beside the columns, not behind them: 0.9 us less a check.
  if (warp == 6 && lane == 0 && flag) out[6] = (double)*(const volatile int*)flag;
  if (tid == 0) *count = 0;
}

void launch_fold(int precision, const GridLaunch& L, const GridGeom& G, const uint8_t* mask,
                 const float* xin, const void* e, float* xout, cudaStream_t st) {
  if (precision == FPIE_MIXED_BF16)
    grid_fold_kernel<<<L.sweep_grid, L.sweep_block, 0, st>>>(
        G, mask, xin, static_cast<const __nv_bfloat16*>(e), xout);
  else
    grid_fold_kernel<<<L.sweep_grid, L.sweep_block, 0, st>>>(
        G, mask, xin, static_cast<const __half*>(e), xout);
}

void launch_norms(const GridLaunch& L, const GridGeom& G, const uint8_t* mask, const float* g,
                  const float* x, double* parts, unsigned* count, double* out, cudaStream_t st,
                  const int* flag) {
  grid_norms_kernel<<<L.finish_grid, L.finish_block, 0, st>>>(G, mask, g, x, parts, count, out,
                                                              flag, L.finish_rows);
}

}  // namespace fpie
