// Shared definitions of the fpie_gb300 CUDA backend: error plumbing, the
// solver handle, and the small device helpers every kernel uses.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>

#include "fpie_gb300.h"

namespace fpie {

// ---- error reporting ------------------------------------------------------
void set_error(const std::string& msg);
void clear_error();

struct Error {
  int code;
  std::string msg;
};

#define FPIE_CUDA(call)                                                     \
  do {                                                                      \
    cudaError_t e_ = (call);                                                \
    if (e_ != cudaSuccess) {                                                \
      throw ::fpie::Error{FPIE_ERR_CUDA, std::string(#call) + ": " +        \
                                             cudaGetErrorString(e_)};       \
    }                                                                       \
  } while (0)

#define FPIE_REQUIRE(cond, code, msg)                   \
  do {                                                  \
    if (!(cond)) throw ::fpie::Error{(code), (msg)};    \
  } while (0)

// Runs `body` and converts exceptions to a status code + last-error string.
template <class F>
int guarded(F&& body) {
  try {
    clear_error();
    body();
    return FPIE_OK;
  } catch (const Error& e) {
    set_error(e.msg);
    return e.code;
  } catch (const std::exception& e) {
    set_error(e.what());
    return FPIE_ERR_STATE;
  }
}

// Blocks for a grid-stride loop over `total` elements, `threads` per block:
// one block per `threads` elements, at most `per_sm` blocks per SM of the
// current device (its multiprocessor count is read once per device), at
// least 1.
int stride_blocks(long long total, int threads, int per_sm);

// Stream-ordered device scratch that is released on every exit path,
// exceptions included (cudaFreeAsync on the stream it was allocated on).
// The library's stream-ordered scratch pool on the current device.  Unlike
// the device's default pool (release threshold 0: freed memory goes back to
// the driver at every synchronize, and the next reset maps it again), it
// keeps up to 4 GiB of freed scratch for reuse.
cudaMemPool_t scratch_pool();

struct AsyncScratch {
  void* ptr = nullptr;
  cudaStream_t stream = nullptr;
  AsyncScratch(size_t bytes, cudaStream_t st) : stream(st) {
    FPIE_CUDA(cudaMallocFromPoolAsync(&ptr, bytes, scratch_pool(), st));
  }
  ~AsyncScratch() {
    if (ptr) cudaFreeAsync(ptr, stream);
  }
  AsyncScratch(const AsyncScratch&) = delete;
  AsyncScratch& operator=(const AsyncScratch&) = delete;
  char* bytes() const { return static_cast<char*>(ptr); }
};

// Arrays that live in one device block, each 256-byte aligned; the first
// `cleared` of them are zeroed together.  An array of no bytes stays NULL.
struct DevicePart {
  void* pointer;  // where the array's pointer is
  size_t bytes;
};
struct DeviceLayout {
  size_t total = 0, clear = 0;
};
inline DeviceLayout device_layout(const DevicePart* parts, int count, int cleared) {
  DeviceLayout l;
  for (int k = 0; k < count; ++k) {
    l.total += (parts[k].bytes + 255) / 256 * 256;
    if (k < cleared) l.clear = l.total;
  }
  return l;
}
inline void device_place(const DevicePart* parts, int count, void* block) {
  char* at = static_cast<char*>(block);
  for (int k = 0; k < count; ++k) {
    if (parts[k].bytes) *static_cast<void**>(parts[k].pointer) = at;
    at += (parts[k].bytes + 255) / 256 * 256;
  }
}

// ---- grid geometry ----------------------------------------------------------
// The grid state lives in HBM as three planar float32 channel planes with a
// zero halo of kPad rows above and kPad columns left of the crop, and
// kPad + slack rows/columns below and right of it.
// Rows are `pitch` floats apart, pitch a multiple of 32 (128 bytes), so the
// first crop column of every row is 16-byte aligned.  The halo lets every
// tile (including its temporal-blocking apron) be read without bounds checks.
constexpr int kPad = 32;

struct GridGeom {
  int n, m;          // crop rows, columns
  int pitch;         // floats per padded row
  int rows;          // n + 2*kPad + kSlackRows
  long long plane;   // floats per channel plane (pitch * rows)
  __host__ __device__ long long at(int i, int j) const {
    return (long long)(i + kPad) * pitch + (j + kPad);
  }
};

// Rows/columns reserved past the crop's far edges beyond kPad, so that the
// last tile of any temporally blocked variant (tile up to 224 rows / 120
// columns plus its apron) reads and writes inside the allocation.
constexpr int kSlackRows = 256;
constexpr int kSlackCols = 128;

inline GridGeom make_geom(int n, int m) {
  GridGeom g;
  g.n = n;
  g.m = m;
  g.pitch = ((m + 2 * kPad + kSlackCols) + 31) / 32 * 32;
  g.rows = n + 2 * kPad + kSlackRows;
  g.plane = (long long)g.pitch * g.rows;
  return g;
}

// Rows per thread of kernels whose threads own 4 columns and go downwards:
// one while the grid has fewer groups of 4 pixels than the device has threads
// (a chain of dependent row loads would be all that such a kernel takes: 14 us
// against 6 with 4 rows on a 152x152 grid), up to 8 beyond.
int rows_per_thread(const GridGeom& g);

// ---- device helpers -----------------------------------------------------------
// The update keeps the numpy backend's evaluation order exactly:
// ((((g + up) + down) + left) + right) * 0.25  (x/4 and x*0.25 round alike).
// __fadd_rn/__fmul_rn are never contracted into FMAs.
__device__ __forceinline__ float jacobi5(float g, float u, float d, float l,
                                         float r) {
  return __fmul_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(g, u), d), l), r),
                   0.25f);
}

// Grid residual in the numpy backend's order: 4x - g - up - down - left - right.
__device__ __forceinline__ float grid_res(float x, float g, float u, float d,
                                          float l, float r) {
  float t = __fsub_rn(__fmul_rn(4.0f, x), g);
  t = __fsub_rn(t, u);
  t = __fsub_rn(t, d);
  t = __fsub_rn(t, l);
  return __fsub_rn(t, r);
}

// Clamp to [0,255] and truncate, as the reference's uint8 store does.
__device__ __forceinline__ uint8_t clip_u8(float v) {
  v = fminf(fmaxf(v, 0.0f), 255.0f);
  return (uint8_t)__float2int_rz(v);
}

__device__ __forceinline__ float4 ld4(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}

// Block-wide sum of three doubles; the result is valid in thread 0.
// blockDim.x * blockDim.y must be a multiple of 32 and at most 1024.
__device__ __forceinline__ void block_sum3(double& a, double& b, double& c) {
  __shared__ double sh[3][32];
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int nwarps = (blockDim.x * blockDim.y) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
    c += __shfl_down_sync(0xffffffffu, c, o);
  }
  if (lane == 0) {
    sh[0][warp] = a;
    sh[1][warp] = b;
    sh[2][warp] = c;
  }
  __syncthreads();
  if (warp == 0) {
    a = lane < nwarps ? sh[0][lane] : 0.0;
    b = lane < nwarps ? sh[1][lane] : 0.0;
    c = lane < nwarps ? sh[2][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
      c += __shfl_down_sync(0xffffffffu, c, o);
    }
  }
}

// A sum of floats as hi + mid + lo (Knuth's error-free addition), exact to
// about 2^-70 of it: more than a sum of doubles keeps, without FP64 adds, which
// run at about two per SM and cycle here.  The blocks' partials and the total
// are doubles.  A finish of a 3603x3603 crop takes 104 us (297 with sums of
// doubles and one row per thread), of 802x802 13.4 (26.4).
struct Sum3 {
  float hi = 0.f, mid = 0.f, lo = 0.f;
};
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float t = __fadd_rn(a, b), c = __fsub_rn(t, a);
  err = __fadd_rn(__fsub_rn(a, __fsub_rn(t, c)), __fsub_rn(b, c));
  return t;
}
__device__ __forceinline__ void sum3_add(Sum3& s, float v) {
  float e, f;
  s.hi = two_sum(s.hi, v, e);
  s.mid = two_sum(s.mid, e, f);
  s.lo = __fadd_rn(s.lo, f);
}
__device__ __forceinline__ void sum3_join(Sum3& s, const Sum3& t) {
  float e;
  sum3_add(s, t.hi);
  s.mid = two_sum(s.mid, t.mid, e);
  s.lo = __fadd_rn(s.lo, __fadd_rn(t.lo, e));
}
// The warp's sum, in lane 0.
__device__ __forceinline__ void sum3_warp(Sum3& s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const Sum3 t{__shfl_down_sync(0xffffffffu, s.hi, o), __shfl_down_sync(0xffffffffu, s.mid, o),
                 __shfl_down_sync(0xffffffffu, s.lo, o)};
    sum3_join(s, t);
  }
}
// The value; where hi overflowed or is no number, hi alone.
__device__ __forceinline__ double sum3_value(const Sum3& s) {
  return isfinite(s.hi) ? ((double)s.hi + (double)s.mid) + (double)s.lo : (double)s.hi;
}

// Block-wide sums of acc[3] to parts[3 * block ...], and by the last block to
// arrive the total of all blocks' parts to err[3], in a fixed order.  256
// threads; every thread of every block calls it.  count: a device word, 0
// before the first launch; the last block clears it.  err may be pinned host
// memory: then no copy follows (3-4 us of a step).  flag, unless NULL, goes to
// err[3] with it.
__device__ __forceinline__ void finish_sums(Sum3 (&acc)[3], unsigned block, unsigned blocks,
                                            double* parts, unsigned* count, float* err,
                                            const int* flag) {
  // Two warps per channel, each from half of the threads' sums: all warps
  // reducing their own three channels was 120 joins a block instead of 48.
  __shared__ Sum3 sums[3][256];
  __shared__ double sh[3][2];
  __shared__ bool last;
  const int tid = threadIdx.x + threadIdx.y * blockDim.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int k = 0; k < 3; ++k) sums[k][tid] = acc[k];
  __syncthreads();
  if (warp < 6) {
    const Sum3* from = sums[warp >> 1] + 128 * (warp & 1) + lane;
    Sum3 s = from[0];
#pragma unroll
    for (int k = 32; k < 128; k += 32) sum3_join(s, from[k]);
    sum3_warp(s);
    if (lane == 0) sh[warp >> 1][warp & 1] = sum3_value(s);
  }
  __syncthreads();
  if (tid < 3) {
    parts[3 * (size_t)block + tid] = sh[tid][0] + sh[tid][1];
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last = atomicAdd(count, 1u) == blocks - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 0.0, b = 0.0, c = 0.0;
  for (unsigned k = tid; k < blocks; k += 256) {
    a += __ldcg(parts + 3 * (size_t)k);
    b += __ldcg(parts + 3 * (size_t)k + 1);
    c += __ldcg(parts + 3 * (size_t)k + 2);
  }
  block_sum3(a, b, c);
  if (tid == 0) {
    err[0] = (float)a;
    err[1] = (float)b;
    err[2] = (float)c;
    if (flag) err[3] = __int_as_float(*(const volatile int*)flag);
    *count = 0;
  }
}

// Sums `nparts` per-block partials (3 doubles each) into err[3] (float) in a
// fixed order, so the result does not depend on block scheduling.
void launch_finalize(const double* parts, int nparts, float* err,
                     cudaStream_t st);

// ---- solver handle -----------------------------------------------------------
struct Solver {
  int kind = 0;  // 1 = equ, 2 = grid
  int device = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;  // where work is enqueued
  long long launches = 0;
  int precision = FPIE_FP32;
  virtual ~Solver() {}
  // The error a kernel recorded in device memory (e.g. a bounded wait that
  // timed out): queue_check queues a copy of it, check_async raises it once the
  // stream has been synchronised.
  virtual void queue_check() {}
  virtual void check_async() {}
  void activate() const { FPIE_CUDA(cudaSetDevice(device)); }
};

Solver* new_equ_solver(int block_size);
Solver* new_grid_solver(int grid_x, int grid_y);

inline Solver* check_handle(fpie_solver* s, int kind) {
  FPIE_REQUIRE(s != nullptr, FPIE_ERR_ARG, "null solver handle");
  Solver* h = reinterpret_cast<Solver*>(s);
  if (kind) FPIE_REQUIRE(h->kind == kind, FPIE_ERR_ARG, "wrong solver kind for this call");
  h->activate();
  return h;
}

// Launch-configuration check: every launch is followed by this, so a bad
// configuration surfaces as an error status at the call that caused it.
inline void post_launch(Solver* s, int n = 1) {
  s->launches += n;
  FPIE_CUDA(cudaGetLastError());
}

}  // namespace fpie
