// The quartered Jacobi sweep on register-resident strips, for the resident
// kernel (grid_res.cu) and the batch (batch.cu).
//
// A pixel's next value is ((((g + up) + down) + left) + right) / 4 in the
// numpy order.  Scaling by 1/4 commutes with rounding, so with g' = g / 4 it
// is fma(right, 1/4, fma(left, 1/4, fma(down, 1/4, fma(up, 1/4, g')))): the
// same bits in four FFMAs instead of four additions and a multiplication.  An
// unmasked pixel keeps its value by one maximum instead of a select on mask
// bits: its g' is -inf, so the sum is -inf, and L, the value to keep, wins; a
// masked pixel's L is a NaN, which a maximum ignores.  (Measured per 128x128
// region and sweep, 8 warps: 690 cycles fully masked, 830-900 with the
// maximum; the packed FADD2 sweep 725, with its selects 1,220.  A packed FADD2
// takes two issue slots, so pairing rows gains nothing and costs register
// moves; a multiplier register per pixel instead of the maximum, 880.)
//
// Where the scaling is exact.  A quartered partial sum that is a multiple of
// 2^-149 is a quarter of the unquartered one, rounded alike: below 2^-126 both
// are exact, above both keep 24 bits.  An unquartered one overflows only above
// 2^127, and -inf + inf is no number.  The kernels therefore
//  (1) read a mark (`wild`) that a reset sets for inputs that are not finite,
//      above 2^40, or (gradients) nonzero below 2^-94, and with it take
//      slow_sweep, the reference's order of operations, throughout.  Bounded
//      inputs stay bounded: a sweep adds at most max|g| / 4.
//  (2) look for nonzero values below 2^-94 every 16 sweeps.  Without any, all
//      values and gradients are multiples of 2^-117; every sweep makes that at
//      most four times finer, so for 16 sweeps partial sums are multiples of
//      2^-149.  With some, the resident kernel keeps the reference's order of
//      additions (QUARTER false: six operations instead of five), the batch
//      its packed update.  Such values are no rarity: on black without a
//      gradient they run ahead of what diffuses into it (255 / 4^k at the k-th
//      pixel), on 802x802 for thousands of sweeps.
#pragma once

#include "common.cuh"

namespace fpie {

constexpr unsigned kMasked = 0x7fffffffu;   // L of a masked pixel (a NaN)
constexpr unsigned kNegInf = 0xff800000u;   // g' of an unmasked pixel
constexpr int kTiny = 94;                   // 2^-kTiny: the limit above

// 2 * |bits| - 1 of v, so that zeros wrap to the top: compare with tiny_limit.
__device__ __forceinline__ unsigned tiny_key(float v) { return 2u * __float_as_uint(v) - 1u; }
constexpr unsigned tiny_limit(int e) { return 2u * ((127u - e) << 23) - 1u; }  // of 2^-e

// The edge rows of a strip, for its neighbours' next sweep.
template <int R, int NS, int LW>
__device__ __forceinline__ void post_edges(const float (&P)[R][4], int par, int lane, int w,
                                           float4 (&edge)[2][2][NS][LW]) {
  edge[par][0][w][lane] = make_float4(P[0][0], P[0][1], P[0][2], P[0][3]);
  edge[par][1][w][lane] = make_float4(P[R - 1][0], P[R - 1][1], P[R - 1][2], P[R - 1][3]);
}

// One in-place sweep of the strip P (R rows x 4 columns per thread, region rows
// w * R on; a strip is LW lanes, half a warp where LW = 16), edge rows through
// shared memory, columns by shuffles.  On entry edge[par] holds the strips'
// edge rows (post_edges and a barrier before the first sweep), on return
// edge[par ^ 1] the new ones, and all strips have read the old.  FWD visits
// rows downwards, !FWD upwards, each keeping the old row it just replaced: a
// forward and a backward sweep leave every row in its registers.  Rows are
// visited in a circle that passes the edge rows in the middle, so that the
// neighbours' rows are loaded behind the first rows' work and the new edge
// rows stored before the last rows' (fully masked region of 8 rows, 4 warps:
// 302 cycles a sweep against 318 from the top row down; through an mbarrier
// with arrival and wait apart, 424).
// FULL: all of the region is masked.  !QUARTER: the reference's order, with
// finite values only (an unmasked pixel's sum has to stay -inf); 4 g' + up
// rounds as g + up does.
template <int R, int NS, int LW, bool FULL, bool FWD, bool QUARTER = true>
__device__ __forceinline__ void quarter_sweep(float (&P)[R][4], const float (&Gq)[R][4],
                                              const float (&L)[FULL ? 1 : R][4], int par, int lane,
                                              int w, float4 (&edge)[2][2][NS][LW]) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 a4 = w > 0 ? edge[par][1][w - 1][lane] : zero;
  const float4 b4 = w < NS - 1 ? edge[par][0][w + 1][lane] : zero;
  const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
  constexpr int F = FWD ? 2 : R - 3;  // the first row visited
  float keep[4], first[4];            // the old rows just replaced, and F
#pragma unroll
  for (int j = 0; j < 4; ++j) first[j] = P[F][j];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int i = FWD ? (F + k) % R : (F - k + R) % R;
    const float cur[4] = {P[i][0], P[i][1], P[i][2], P[i][3]};
    const float lf = __shfl_up_sync(0xffffffffu, cur[3], 1, LW);
    const float rt = __shfl_down_sync(0xffffffffu, cur[0], 1, LW);
    float t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float up = i == 0                 ? a[j]
                       : FWD && k > 0         ? keep[j]
                       : !FWD && k == R - 1   ? first[j]
                                              : P[i > 0 ? i - 1 : 0][j];
      t[j] = QUARTER ? __fmaf_rn(up, 0.25f, Gq[i][j]) : __fmaf_rn(Gq[i][j], 4.f, up);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float down = i == R - 1             ? b[j]
                         : !FWD && k > 0        ? keep[j]
                         : FWD && k == R - 1    ? first[j]
                                                : P[i < R - 1 ? i + 1 : i][j];
      t[j] = QUARTER ? __fmaf_rn(down, 0.25f, t[j]) : __fadd_rn(t[j], down);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float left = j > 0 ? cur[j > 0 ? j - 1 : 0] : lf;
      t[j] = QUARTER ? __fmaf_rn(left, 0.25f, t[j]) : __fadd_rn(t[j], left);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      keep[j] = cur[j];
      const float right = j < 3 ? cur[j < 3 ? j + 1 : 0] : rt;
      const float o = QUARTER ? __fmaf_rn(right, 0.25f, t[j])
                              : __fmul_rn(__fadd_rn(t[j], right), 0.25f);
      P[i][j] = FULL ? o : fmaxf(o, L[FULL ? 0 : i][j]);
    }
    if (i == (FWD ? 0 : R - 1)) post_edges<R, NS, LW>(P, par ^ 1, lane, w, edge);
  }
  __syncthreads();
}

// The same sweep in the reference's order of operations, for any values and
// for a single sweep: gs * G is the gradient (gs 4, or 1 where G is
// not quartered), `on(i, j)` tells the masked pixels.
template <int R, int NS, int LW, typename On>
__device__ __forceinline__ void slow_sweep(float (&P)[R][4], const float (&G)[R][4], On on,
                                           float gs, int lane, int w,
                                           float4 (&edge)[2][2][NS][LW]) {
  post_edges<R, NS, LW>(P, 0, lane, w, edge);
  __syncthreads();
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 a4 = w > 0 ? edge[0][1][w - 1][lane] : zero;
  const float4 b4 = w < NS - 1 ? edge[0][0][w + 1][lane] : zero;
  const float b[4] = {b4.x, b4.y, b4.z, b4.w};
  float keep[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float cur[4] = {P[i][0], P[i][1], P[i][2], P[i][3]};
    const float lf = __shfl_up_sync(0xffffffffu, cur[3], 1, LW);
    const float rt = __shfl_down_sync(0xffffffffu, cur[0], 1, LW);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float o = jacobi5(__fmul_rn(G[i][j], gs), keep[j],
                              i < R - 1 ? P[i < R - 1 ? i + 1 : i][j] : b[j],
                              j > 0 ? cur[j > 0 ? j - 1 : 0] : lf, j < 3 ? cur[j < 3 ? j + 1 : 0] : rt);
      keep[j] = cur[j];
      if (on(i, j)) P[i][j] = o;
    }
  }
  __syncthreads();  // the edge rows are read before the next sweep writes them
}

}  // namespace fpie
