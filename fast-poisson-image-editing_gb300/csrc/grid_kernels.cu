// Grid sweep and finish kernels (FP32, one sweep per launch).
//
// Each thread owns four horizontally adjacent pixels of one row (one float4
// per channel plane).  A warp covers 128 consecutive columns, so every
// plane access is a 512-byte coalesced run; the left/right neighbours of the
// group's end pixels come from two scalar loads that hit the same L1 lines.
// Groups with no masked pixel do nothing: their values never change and both
// state buffers already hold them.
#include "grid_kernels.cuh"

namespace fpie {

constexpr int kSweepBX = 64, kSweepBY = 4;

__global__ void __launch_bounds__(kSweepBX * kSweepBY)
grid_sweep_kernel(GridGeom G, const uint8_t* __restrict__ mask,
                  const float* __restrict__ g, const float* __restrict__ xin,
                  float* __restrict__ xout) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;  // 4-column group
  const int i = blockIdx.y * blockDim.y + threadIdx.y;  // crop row
  if (i >= G.n || 4 * q >= G.m) return;
  const long long p = G.at(i, 4 * q);
  const uint32_t mk = *reinterpret_cast<const uint32_t*>(mask + p);
  if (mk == 0u) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float* xc = xin + c * G.plane;
    const float4 ce = ld4(xc + p);
    const float4 up = ld4(xc + p - G.pitch);
    const float4 dn = ld4(xc + p + G.pitch);
    const float lf = __ldg(xc + p - 1);
    const float rt = __ldg(xc + p + 4);
    const float4 gg = ld4(g + c * G.plane + p);
    float4 o;
    o.x = (mk & 0x000000ffu) ? jacobi5(gg.x, up.x, dn.x, lf, ce.y) : ce.x;
    o.y = (mk & 0x0000ff00u) ? jacobi5(gg.y, up.y, dn.y, ce.x, ce.z) : ce.y;
    o.z = (mk & 0x00ff0000u) ? jacobi5(gg.z, up.z, dn.z, ce.y, ce.w) : ce.z;
    o.w = (mk & 0xff000000u) ? jacobi5(gg.w, up.w, dn.w, ce.z, rt) : ce.w;
    *reinterpret_cast<float4*>(xout + c * G.plane + p) = o;
  }
}

// Stores the 12 bytes w0 w1 w2 of each lane's four pixels to `a` + 12 * lane
// (a: the warp's first byte, any alignment) as aligned words: a lane's words
// take the last bytes of the lane before it.  n: this lane's pixels (0-4; only
// the last lane of a row has 1-3).  Byte stores of all 12 took most of a
// finish's store time.
__device__ __forceinline__ void store_run(uint8_t* a, unsigned w0, unsigned w1, unsigned w2,
                                          int n) {
  const int lane = threadIdx.x & 31;
  const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(a) & 3), sh = 8 * s;
  const unsigned before = __shfl_up_sync(0xffffffffu, w2, 1);
  const int after = __shfl_down_sync(0xffffffffu, n, 1);
  uint8_t* const p = a + 12 * lane;
  if (n == 4) {
    unsigned* const q = reinterpret_cast<unsigned*>(p - s);
    if (lane > 0 || s == 0)
      q[0] = __funnelshift_l(before, w0, sh);
    else
      for (unsigned k = 0; k < 4 - s; ++k) p[k] = (uint8_t)(w0 >> (8 * k));
    q[1] = __funnelshift_l(w0, w1, sh);
    q[2] = __funnelshift_l(w1, w2, sh);
    if (lane == 31 || after != 4)  // nobody else stores this lane's last s bytes
      for (unsigned k = 0; k < s; ++k) p[12 - s + k] = (uint8_t)(w2 >> (8 * (4 - s + k)));
  } else {
    const unsigned w[3] = {w0, w1, w2};
#pragma unroll
    for (int k = 0; k < 9; ++k)
      if (k < 3 * n) p[k] = (uint8_t)(w[k / 4] >> (8 * (k % 4)));
  }
}

// Thread: four columns, `rows` rows downwards (rows_per_thread).  Measured on
// a 3603x3603 crop: 103 us; 240 with a row per thread, byte stores and FP64
// sums.

__global__ void __launch_bounds__(kSweepBX * kSweepBY)
grid_finish_kernel(GridGeom G, const uint8_t* __restrict__ mask,
                   const float* __restrict__ g, const float* __restrict__ x,
                   uint8_t* __restrict__ img, double* __restrict__ parts,
                   unsigned* __restrict__ count, float* __restrict__ err,
                   const int* flag, int rows) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int i0 = (blockIdx.y * blockDim.y + threadIdx.y) * rows;
  Sum3 acc[3];
  const int jn = max(0, min(4, G.m - 4 * q));
  const int i1 = min(i0 + rows, G.n);
  for (int i = i0; i < i1; ++i) {  // uniform per warp
    unsigned w0 = 0, w1 = 0, w2 = 0;
    if (jn > 0) {
      const long long p = G.at(i, 4 * q);
      const uint32_t mk = __ldg(reinterpret_cast<const uint32_t*>(mask + p));
      unsigned b[12];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float* xc = x + c * G.plane;
        const float4 ce = ld4(xc + p);
        if (mk) {
          const float4 up = ld4(xc + p - G.pitch);
          const float4 dn = ld4(xc + p + G.pitch);
          const float lf = __ldg(xc + p - 1);
          const float rt = __ldg(xc + p + 4);
          const float4 gg = ld4(g + c * G.plane + p);
          // Per-pixel |r| is exact float32 (numpy order).
          if (mk & 0x000000ffu) sum3_add(acc[c], fabsf(grid_res(ce.x, gg.x, up.x, dn.x, lf, ce.y)));
          if (mk & 0x0000ff00u) sum3_add(acc[c], fabsf(grid_res(ce.y, gg.y, up.y, dn.y, ce.x, ce.z)));
          if (mk & 0x00ff0000u) sum3_add(acc[c], fabsf(grid_res(ce.z, gg.z, up.z, dn.z, ce.y, ce.w)));
          if (mk & 0xff000000u) sum3_add(acc[c], fabsf(grid_res(ce.w, gg.w, up.w, dn.w, ce.z, rt)));
        }
        b[c] = clip_u8(ce.x);
        b[3 + c] = clip_u8(ce.y);
        b[6 + c] = clip_u8(ce.z);
        b[9 + c] = clip_u8(ce.w);
      }
      w0 = b[0] | b[1] << 8 | b[2] << 16 | b[3] << 24;
      w1 = b[4] | b[5] << 8 | b[6] << 16 | b[7] << 24;
      w2 = b[8] | b[9] << 8 | b[10] << 16 | b[11] << 24;
    }
    const int q0 = q & ~31;  // the warp's first group
    store_run(img + ((long long)i * G.m + 4 * q0) * 3, w0, w1, w2, jn);
  }
  finish_sums(acc, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y, parts, count, err,
              flag);
}

GridLaunch grid_launch(const GridGeom& G) {
  GridLaunch L;
  const int groups = (G.m + 3) / 4;
  L.sweep_block = dim3(kSweepBX, kSweepBY);
  L.sweep_grid = dim3((groups + kSweepBX - 1) / kSweepBX, (G.n + kSweepBY - 1) / kSweepBY);
  L.finish_block = L.sweep_block;
  L.finish_rows = rows_per_thread(G);
  const int by = kSweepBY * L.finish_rows;
  L.finish_grid = dim3(L.sweep_grid.x, (G.n + by - 1) / by);
  L.nparts = (int)(L.sweep_grid.x * L.sweep_grid.y);
  return L;
}

void launch_grid_sweep(const GridLaunch& L, const GridGeom& G,
                       const uint8_t* mask, const float* g, const float* xin,
                       float* xout, cudaStream_t st) {
  grid_sweep_kernel<<<L.sweep_grid, L.sweep_block, 0, st>>>(G, mask, g, xin, xout);
}

void launch_grid_finish(const GridLaunch& L, const GridGeom& G,
                        const uint8_t* mask, const float* g, const float* x,
                        uint8_t* img, double* parts, unsigned* count, float* err,
                        cudaStream_t st, const int* flag) {
  grid_finish_kernel<<<L.finish_grid, L.finish_block, 0, st>>>(G, mask, g, x, img, parts, count,
                                                               err, flag, L.finish_rows);
}

}  // namespace fpie
