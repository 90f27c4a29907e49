// GPU-side construction of the grid solver's inputs from the three images.
//
// Same results as the host path (GridProcessor.reset, fpie/process.py:321-386),
// bit for bit:
//   * mask: a 3-channel mask is "on" when its channel mean is >= 128, i.e.
//     when the channel sum is >= 384 (exact for uint8); a 1-channel mask when
//     its value is >= 128; the outer 1-pixel frame is cleared;
//   * crop: the set pixels' bounding box grown by one pixel;
//   * grad: for every set pixel, mix(C-U) + mix(C-D) + mix(C-L) + mix(C-R)
//     accumulated from 0 in that order, where mix is 'src' (a), 'avg'
//     ((a+b)/2) or 'max' (b if |a| < |b| else a), a the source difference
//     and b the target difference, all in float32 (every intermediate is a
//     small integer or half-integer, so the sums are exact); 0 elsewhere.
// The outputs go straight into the solver's planar padded layout.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "prep.cuh"

namespace fpie {

// One set of atomics per block and 16 pixels per thread: with a pixel per
// thread and four atomics per warp it took 41 us on a 1024x1024 mask, all of
// it atomics on the same four words (now 4).
// The accumulators are maxima that start at 0 (INT_MAX - row min, row max + 1,
// the same for columns); the last block writes the box and clears them.
template <int CH>
__global__ void __launch_bounds__(256)
prep_mask_kernel(const uint8_t* __restrict__ mask, int mh, int mw, bool aligned,
                 uint8_t* __restrict__ m01, int* __restrict__ acc, int* __restrict__ box) {
  int top = 0, bottom = 0, left = 0, right = 0;
  auto see = [&](int i, int j0, int j1) {
    top = max(top, INT_MAX - i);
    bottom = max(bottom, i + 1);
    left = max(left, INT_MAX - j0);
    right = max(right, j1 + 1);
  };
  const long long total = (long long)mh * mw;
  for (long long p0 = 16 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); p0 < total;
       p0 += 16LL * gridDim.x * blockDim.x) {
    const int cnt = (int)min(16LL, total - p0);
    unsigned on = 0;  // bit k: pixel p0 + k is selected
    if (cnt == 16 && aligned) {
      unsigned v[4 * CH];
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(mask + p0 * CH) + k);
        v[4 * k] = u.x, v[4 * k + 1] = u.y, v[4 * k + 2] = u.z, v[4 * k + 3] = u.w;
      }
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        int sum = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) sum += (v[(k * CH + c) / 4] >> (8 * ((k * CH + c) % 4))) & 0xffu;
        on |= (unsigned)(sum >= 128 * CH) << k;
      }
    } else {
      for (int k = 0; k < cnt; ++k) {
        int sum = 0;
        for (int c = 0; c < CH; ++c) sum += mask[(p0 + k) * CH + c];
        on |= (unsigned)(sum >= 128 * CH) << k;
      }
    }
    int i = (int)(p0 / mw), j = (int)(p0 - (long long)i * mw);
    if (j + cnt <= mw) {  // one row
      if (i == 0 || i == mh - 1) on = 0;
      if (j == 0) on &= ~1u;
      if (j + cnt == mw) on &= ~(1u << (cnt - 1));
      if (on) see(i, j + __ffs(on) - 1, j + 31 - __clz(on));
    } else {
      for (int k = 0; k < cnt; ++k) {
        if (i == 0 || i == mh - 1 || j == 0 || j == mw - 1) on &= ~(1u << k);
        if ((on >> k) & 1u) see(i, j, j);
        if (++j == mw) {
          j = 0;
          ++i;
        }
      }
    }
    if (cnt == 16) {  // bits to bytes, four at a time
      uint4 o;
      o.x = ((on & 15u) * 0x00204081u) & 0x01010101u;
      o.y = (((on >> 4) & 15u) * 0x00204081u) & 0x01010101u;
      o.z = (((on >> 8) & 15u) * 0x00204081u) & 0x01010101u;
      o.w = ((on >> 12) * 0x00204081u) & 0x01010101u;
      *reinterpret_cast<uint4*>(m01 + p0) = o;
    } else {
      for (int k = 0; k < cnt; ++k) m01[p0 + k] = (on >> k) & 1u;
    }
  }
  __shared__ int sh[4];
  __shared__ bool last;
  if (threadIdx.x < 4) sh[threadIdx.x] = 0;
  __syncthreads();
  const int v[4] = {top, bottom, left, right};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int m = __reduce_max_sync(0xffffffffu, v[k]);
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(&sh[k], m);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (sh[1] > 0)
      for (int k = 0; k < 4; ++k) atomicMax(acc + k, sh[k]);
    __threadfence();
    last = atomicAdd(acc + 4, 1) == (int)gridDim.x - 1;
    if (last) {
      __threadfence();
      const int r = atomicExch(acc + 0, 0), r1 = atomicExch(acc + 1, 0);
      const int c = atomicExch(acc + 2, 0), c1 = atomicExch(acc + 3, 0);
      acc[4] = 0;
      box[0] = r1 ? INT_MAX - r : INT_MAX;
      box[1] = r1 - 1;
      box[2] = r1 ? INT_MAX - c : INT_MAX;
      box[3] = c1 - 1;
    }
  }
}

// The mixed term in integers: twice the mean for 'avg' (every term and sum is
// an integer or a half below 2^11, so the float32 sums are these, scaled).
__device__ __forceinline__ int mix_int(int a, int b, int mode) {
  if (mode == 0) return a;
  if (mode == 1) return a + b;
  return abs(a) < abs(b) ? b : a;
}

// 6 pixels (18 bytes) of an image row from byte `a` on, as 5 words, of which
// the bytes in [lo, hi) are used.  Words are read where all of them lie in the
// image [im, end), bytes at its first and last pixels.
__device__ __forceinline__ void load_px6(const uint8_t* a, const uint8_t* lo, const uint8_t* hi,
                                         const uint8_t* im, const uint8_t* end, unsigned (&o)[5]) {
  const unsigned sh = 8 * (unsigned)(reinterpret_cast<uintptr_t>(a) & 3);
  const uint8_t* w = a - (sh >> 3);
  unsigned v[6];
  if (w >= im && w + 24 <= end) {
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = __ldg(reinterpret_cast<const unsigned*>(w + 4 * k));
  } else {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      v[k] = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const uint8_t* p = w + 4 * k + b;
        if (p >= lo && p < hi) v[k] |= (unsigned)__ldg(p) << (8 * b);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) o[k] = __funnelshift_r(v[k], v[k + 1], sh);
}

__device__ __forceinline__ int px_byte(const unsigned (&w)[5], int b) {
  return (int)((w[b / 4] >> (8 * (b % 4))) & 0xffu);
}

// Thread: 4 adjacent columns, `rows` rows downwards, so that a row of either
// image is read once for itself and its two neighbours, as words.  (With one
// pixel per thread, 30 byte loads each, it took 155 us on a 3603x3603 crop.)

__global__ void __launch_bounds__(256)
prep_grid_kernel(PrepArgs A, uint8_t* __restrict__ mask, float* __restrict__ xa,
                 float* __restrict__ xb, float* __restrict__ g, int rows) {
  const GridGeom& G = A.G;
  const int j0 = 4 * (blockIdx.x * 64 + (threadIdx.x & 63));
  const int i0 = (blockIdx.y * 4 + (threadIdx.x >> 6)) * rows;
  if (j0 >= G.m || i0 >= G.n) return;
  const int cl = max(j0 - 1, 0), cr = min(j0 + 5, G.m);  // crop columns read
  auto row = [&](const uint8_t* im, int h, int w, int r0, int c0, int i, unsigned (&o)[5]) {
    const uint8_t* p = im + ((long long)(r0 + i) * w + c0) * 3;
    load_px6(p + 3 * (j0 - 1), p + 3 * cl, p + 3 * cr, im, im + (long long)h * w * 3, o);
  };
  unsigned su[5] = {}, sc[5], sd[5] = {}, tu[5] = {}, tc[5], td[5] = {};
  if (i0 > 0) {
    row(A.src, A.sh, A.sw, A.sx, A.sy, i0 - 1, su);
    row(A.tgt, A.th, A.tw, A.tx, A.ty, i0 - 1, tu);
  }
  row(A.src, A.sh, A.sw, A.sx, A.sy, i0, sc);
  row(A.tgt, A.th, A.tw, A.tx, A.ty, i0, tc);
  const int i1 = min(i0 + rows, G.n);
  const float scale = A.mode == 1 ? 0.5f : 1.0f;
  for (int i = i0; i < i1; ++i) {
    if (i + 1 < G.n) {
      row(A.src, A.sh, A.sw, A.sx, A.sy, i + 1, sd);
      row(A.tgt, A.th, A.tw, A.tx, A.ty, i + 1, td);
    }
    const uint8_t* mr = A.m01 + (long long)(A.x0 + i) * A.mw + A.y0 + j0;
    unsigned on = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j0 + k < G.m && mr[k]) on |= 1u << (8 * k);
    const long long p = G.at(i, j0);
    *reinterpret_cast<unsigned*>(mask + p) = on;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float t[4], r[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int b = 3 * (k + 1) + c;
        const int s0 = px_byte(sc, b), t0 = px_byte(tc, b);
        t[k] = j0 + k < G.m ? (float)t0 : 0.f;
        // Set pixels are never on the crop border: all 4 neighbours exist.
        int acc = mix_int(s0 - px_byte(su, b), t0 - px_byte(tu, b), A.mode);
        acc += mix_int(s0 - px_byte(sd, b), t0 - px_byte(td, b), A.mode);
        acc += mix_int(s0 - px_byte(sc, b - 3), t0 - px_byte(tc, b - 3), A.mode);
        acc += mix_int(s0 - px_byte(sc, b + 3), t0 - px_byte(tc, b + 3), A.mode);
        r[k] = (on >> (8 * k)) & 1u ? __fmul_rn((float)acc, scale) : 0.f;
      }
      const float4 t4 = make_float4(t[0], t[1], t[2], t[3]);
      *reinterpret_cast<float4*>(xa + c * G.plane + p) = t4;
      *reinterpret_cast<float4*>(xb + c * G.plane + p) = t4;
      *reinterpret_cast<float4*>(g + c * G.plane + p) = make_float4(r[0], r[1], r[2], r[3]);
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      su[k] = sc[k], sc[k] = sd[k];
      tu[k] = tc[k], tc[k] = td[k];
    }
  }
}

void launch_prep_mask(const uint8_t* mask, int mh, int mw, int mch, uint8_t* m01, int* acc,
                      int* box, cudaStream_t st) {
  const long long total = (long long)mh * mw;
  const int blocks = stride_blocks((total + 15) / 16, 256, 8);
  const bool aligned = (reinterpret_cast<uintptr_t>(mask) & 15) == 0;
  if (mch == 3)
    prep_mask_kernel<3><<<blocks, 256, 0, st>>>(mask, mh, mw, aligned, m01, acc, box);
  else
    prep_mask_kernel<1><<<blocks, 256, 0, st>>>(mask, mh, mw, aligned, m01, acc, box);
}

void launch_prep_grid(const PrepArgs& a, uint8_t* mask, float* xa, float* xb, float* g,
                      cudaStream_t st) {
  const int rows = rows_per_thread(a.G);
  const dim3 blocks((a.G.m + 255) / 256, (a.G.n + 4 * rows - 1) / (4 * rows));
  prep_grid_kernel<<<blocks, 256, 0, st>>>(a, mask, xa, xb, g, rows);
}

}  // namespace fpie

// ---- equation form ---------------------------------------------------------------
// ids: 1-based row-major ranks of the set pixels of the crop (the reference's
// partition + ids[mask == 0] = 0, fpie/process.py:180-190), by a three-step
// scan over blocks of kScanTile pixels.  Red-black numbering (the OpenMP
// EquSolver's partition, fpie/core/openmp/equ.cc:22-56): the same scan over
// the cells with odd row + col of the crop, then over the even ones, whose
// ranks continue after the odd count.
namespace fpie {

constexpr int kScanTile = 1024;  // 256 threads x 4 pixels

struct CropView {
  const uint8_t* m01;
  int mw, x0, y0, n, m;
  int parity = -1;  // 0 / 1: only the cells with that parity of row + col count as set
  __device__ __forceinline__ int at(long long q) const {
    const int i = (int)(q / m), j = (int)(q % m);
    if (parity >= 0 && ((i + j) & 1) != parity) return 0;
    return m01[(long long)(x0 + i) * mw + (y0 + j)];
  }
};

__global__ void __launch_bounds__(256) scan_count_kernel(CropView V, int* __restrict__ counts) {
  const long long total = (long long)V.n * V.m;
  const long long start = (long long)blockIdx.x * kScanTile;
  int c = 0;
  for (int k = threadIdx.x; k < kScanTile; k += blockDim.x)
    if (start + k < total) c += V.at(start + k) != 0;
  __shared__ int warp_sum[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < 8; ++w) s += warp_sum[w];
    counts[blockIdx.x] = s;
  }
}

// One block: exclusive scan of the block counts in place; total at counts[nb].
__global__ void __launch_bounds__(1024) scan_offsets_kernel(int* __restrict__ counts, int nb) {
  __shared__ int carry;
  __shared__ int sh[1024];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < nb; base += 1024) {
    const int k = base + threadIdx.x;
    const int v = k < nb ? counts[k] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {  // inclusive Hillis-Steele scan
      const int t = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += t;
      __syncthreads();
    }
    if (k < nb) counts[k] = carry + sh[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += sh[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) counts[nb] = carry;
}

// base: added to every rank (NULL: 0); keep_others: leave the ids of cells
// that do not count as set (second pass of the red-black numbering).
__global__ void __launch_bounds__(256) scan_ids_kernel(CropView V, const int* __restrict__ offsets,
                                                      int* __restrict__ ids,
                                                      const int* __restrict__ base,
                                                      bool keep_others) {
  const long long total = (long long)V.n * V.m;
  const long long start = (long long)blockIdx.x * kScanTile + threadIdx.x * 4;
  int on[4], c = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    on[k] = start + k < total ? V.at(start + k) != 0 : 0;
    c += on[k];
  }
  // exclusive scan of c over the block
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __shared__ int warp_tot[8];
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  int before = 0;
  for (int k = 0; k < w; ++k) before += warp_tot[k];
  int rank = (base ? *base : 0) + offsets[blockIdx.x] + before + incl - c;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (start + k < total && (on[k] || !keep_others)) ids[start + k] = on[k] ? ++rank : 0;
}

// counts[nb] = odd + even unknowns, counts[nb + 1] = odd ones.
__global__ void rb_total_kernel(int* counts, int nb) { counts[nb] += counts[nb + 1]; }

struct EquPrepArgs {
  CropView V;
  const int* ids;  // crop-sized
  const uint8_t* src;
  int sw, sx, sy;
  const uint8_t* tgt;
  int tw, tx, ty;
  int mode;
  long long np;    // plane stride of X/B
};

__device__ __forceinline__ float mix_term2(float a, float b, int mode) {
  if (mode == 0) return a;
  if (mode == 1) return __fmul_rn(__fadd_rn(a, b), 0.5f);
  return fabsf(a) < fabsf(b) ? b : a;
}

// Row id of every set pixel: A = ids of (up, down, left, right), X = target,
// B = grad (L, R, U, D order) + target values of unset neighbours (U, L, R,
// D order), and the pixel's target coordinates (fpie/process.py:227-269).
__global__ void equ_build_kernel(EquPrepArgs P, int4* __restrict__ A, float* __restrict__ x0,
                                 float* __restrict__ x1, float* __restrict__ b,
                                 int* __restrict__ rows, int* __restrict__ cols) {
  const CropView& V = P.V;
  const long long total = (long long)V.n * V.m;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.x * blockDim.x) {
    const int id = P.ids[q];
    if (!id) continue;
    const int i = (int)(q / V.m), j = (int)(q % V.m);
    // set pixels are never on the crop border: all four neighbours exist
    const int iu = P.ids[q - V.m], idn = P.ids[q + V.m], il = P.ids[q - 1], ir = P.ids[q + 1];
    A[id] = make_int4(iu, idn, il, ir);
    rows[id - 1] = P.tx + i;
    cols[id - 1] = P.ty + j;
    const long long sc = ((long long)(P.sx + i) * P.sw + (P.sy + j)) * 3;
    const long long tc = ((long long)(P.tx + i) * P.tw + (P.ty + j)) * 3;
    const long long srow = (long long)P.sw * 3, trow = (long long)P.tw * 3;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float s0 = (float)P.src[sc + c], t0 = (float)P.tgt[tc + c];
      const float tu = P.tgt[tc - trow + c], td = P.tgt[tc + trow + c];
      const float tl = P.tgt[tc - 3 + c], tr = P.tgt[tc + 3 + c];
      float gsum = __fadd_rn(mix_term2(s0 - P.src[sc - 3 + c], t0 - tl, P.mode),
                             mix_term2(s0 - P.src[sc + 3 + c], t0 - tr, P.mode));
      gsum = __fadd_rn(gsum, mix_term2(s0 - P.src[sc - srow + c], t0 - tu, P.mode));
      gsum = __fadd_rn(gsum, mix_term2(s0 - P.src[sc + srow + c], t0 - td, P.mode));
      float bv = gsum;
      if (!iu) bv = __fadd_rn(bv, tu);
      if (!il) bv = __fadd_rn(bv, tl);
      if (!ir) bv = __fadd_rn(bv, tr);
      if (!idn) bv = __fadd_rn(bv, td);
      x0[c * P.np + id] = t0;
      x1[c * P.np + id] = t0;
      b[c * P.np + id] = bv;
    }
  }
}

int launch_equ_ids(const uint8_t* m01, int mw, int x0, int y0, int n, int m, int* counts,
                   int* ids, cudaStream_t st, bool red_black) {
  CropView V{m01, mw, x0, y0, n, m};
  const long long total = (long long)n * m;
  const int nb = (int)((total + kScanTile - 1) / kScanTile);
  if (!red_black) {
    scan_count_kernel<<<nb, 256, 0, st>>>(V, counts);
    scan_offsets_kernel<<<1, 1024, 0, st>>>(counts, nb);
    scan_ids_kernel<<<nb, 256, 0, st>>>(V, counts, ids, nullptr, false);
    return nb;
  }
  V.parity = 1;  // odd cells: ids 1.., every other cell 0
  scan_count_kernel<<<nb, 256, 0, st>>>(V, counts);
  scan_offsets_kernel<<<1, 1024, 0, st>>>(counts, nb);
  scan_ids_kernel<<<nb, 256, 0, st>>>(V, counts, ids, nullptr, false);
  FPIE_CUDA(cudaMemcpyAsync(counts + nb + 1, counts + nb, sizeof(int), cudaMemcpyDeviceToDevice, st));
  V.parity = 0;  // even cells: ids after the odd count
  scan_count_kernel<<<nb, 256, 0, st>>>(V, counts);
  scan_offsets_kernel<<<1, 1024, 0, st>>>(counts, nb);
  scan_ids_kernel<<<nb, 256, 0, st>>>(V, counts, ids, counts + nb + 1, true);
  rb_total_kernel<<<1, 1, 0, st>>>(counts, nb);
  return nb;
}

void launch_equ_build(const uint8_t* m01, int mw, int x0, int y0, int n, int m, const int* ids,
                      const uint8_t* src, int sw, int sx, int sy, const uint8_t* tgt, int tw,
                      int tx, int ty, int mode, long long np, int4* A, float* xa, float* xb,
                      float* b, int* rows, int* cols, cudaStream_t st) {
  EquPrepArgs P{{m01, mw, x0, y0, n, m}, ids, src, sw, sx, sy, tgt, tw, tx, ty, mode, np};
  const long long total = (long long)n * m;
  const int blocks = stride_blocks(total, 256, 32);
  equ_build_kernel<<<blocks, 256, 0, st>>>(P, A, xa, xb, b, rows, cols);
}

}  // namespace fpie
