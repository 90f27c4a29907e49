// Resident grid sweep: one launch per step, one CTA per (tile, channel), all
// co-resident; a tile's state and gradient stay in registers from the first
// sweep to the last, and only the K-pixel ring around it is exchanged with the
// neighbouring tiles, every K sweeps.
//
// What bounds small grids elsewhere is the time between launches or levels
// (a 194x194 grid: 5.6 us per 8-sweep launch, of which ~1.6 us are sweeps):
// launch, region load and store, tail.  Here that is one exchange, and
// regions are cut as small as lets every SM hold one.  Per sweep: 194x194
// 0.266 us (0.71 as launches of 8 sweeps), 251x389 0.385 (0.83), 176x1457
// 0.523 (0.83).
//
// The update is quarter.cuh's.  Each CTA looks for values below 2^-94 every
// 16 sweeps, before an exchange if there is one; one that finds some takes
// unquartered sweeps until its next look and marks the packets it sends, and a
// CTA that receives a marked packet does the same.
//
// Exchange.  A packet is 16 bytes, three values and an epoch, in one 128-bit
// store: the reader polls the packet itself, so data and readiness arrive
// together (one way 450-850 cycles as the poll falls, against 1,490 with
// release and acquire), without a fence, a flag or a barrier on the sender's
// side.  What bounds an exchange is the volume, all CTAs' packets at once:
// with two values and two epochs in 16 bytes, 194x194 took 0.296 us per sweep
// instead of 0.266 and 660x660 0.716 instead of 0.645.  A tile's packets lie
// together, ordered by the parts of its ring
// that different neighbours read.  Two buffers alternate.
// Overwriting one is safe: a CTA sends exchange p only after it received
// every neighbour's exchange p - 1, which that neighbour sent after reading
// exchange p - 2.  Epochs grow from launch to launch (the last CTA to leave
// advances the base in ctl), so nothing is cleared between launches.
//
// All CTAs of the cooperative launch are co-resident, so waits end; they are
// bounded all the same (spin_limit): past it a CTA records an error, all
// CTAs stop at their next wait, and the host reports FPIE_ERR_TIMEOUT.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "grid_res.cuh"
#include "quarter.cuh"

namespace fpie {

namespace {

struct ResArgs {
  GridGeom G;
  const uint8_t* mask;
  const float* g;
  const float* xin;
  float* xout;
  uint4* packets;  // [2][CTA][packets of a tile]
  unsigned* act;                // [tiles * 3] activity words
  unsigned* ctl;                // [0] epoch base, [1] CTAs that left
  const unsigned* wild;
  int* error;
  int* host_error;
  long long spin_limit;
  // Host or device: the residual maxima of xin; nothing is done if they are
  // within tol.  NULL: none.
  const double* maxima;
  double tol;
  int tiles_x, tiles, sweeps;
};

constexpr int kCheck = 16;  // sweeps between looks for tiny values (quarter.cuh)

// 128-bit relaxed accesses are single transactions.
__device__ __forceinline__ void st_packet(uint4* p, float a, float b, float c, unsigned e) {
  const unsigned long long lo = __float_as_uint(a) | (unsigned long long)__float_as_uint(b) << 32,
                           hi = __float_as_uint(c) | (unsigned long long)e << 32;
  asm volatile(
      "{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }"
      :
      : "l"(p), "l"(lo), "l"(hi)
      : "memory");
}

__device__ __forceinline__ ulonglong2 ld_packet(const uint4* p) {
  ulonglong2 v;
  asm volatile(
      "{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
      : "=l"(v.x), "=l"(v.y)
      : "l"(p)
      : "memory");
  return v;
}

// The thread index, read anew: what is computed from it does not stay in
// registers across the sweeps.
__device__ __forceinline__ int fresh_tid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// The ring of a TH x TW tile, its K outermost pixels, cut into the blocks that
// different neighbours read: three bands of rows (one where TH is K) by three
// of columns, without the middle.  A block's pixels, row by row, fill packets
// of three; the last one repeats the last pixel.
template <int K, int TH, int TW>
struct Ring {
  static constexpr int bands = TH == K ? 1 : 3, last = bands - 1;
  static_assert((TH == K || TH >= 2 * K) && TW >= 2 * K, "bands");
  static constexpr int row0(int i) { return i == 0 ? 0 : i == 1 ? K : TH - K; }
  static constexpr int rows(int i) { return i == 1 ? TH - 2 * K : K; }
  static constexpr int col0(int j) { return j == 0 ? 0 : j == 1 ? K : TW - K; }
  static constexpr int cols(int j) { return j == 1 ? TW - 2 * K : K; }
  static constexpr int count(int i, int j) {  // packets of a block
    return i == 1 && j == 1 ? 0 : (rows(i) * cols(j) + 2) / 3;
  }
  static constexpr int first(int i, int j) {
    int n = 0;
    for (int k = 0; k < 3 * i + j; ++k) n += count(k / 3, k % 3);
    return n;
  }
  static constexpr int packets = first(bands - 1, 3);
  // The block rows [i0, i1) and columns [j0, j1) that the tile to the south
  // (dy 1), north (-1), east (dx 1) or west of this one reads.
  static constexpr int i0(int dy) { return dy > 0 ? last : 0; }
  static constexpr int i1(int dy) { return dy < 0 ? 1 : bands; }
  static constexpr int j0(int dx) { return dx > 0 ? 2 : 0; }
  static constexpr int j1(int dx) { return dx < 0 ? 1 : 3; }
  static constexpr int apron() {  // packets that a tile reads
    int n = 0;
    for (int k = 0; k < 9; ++k)
      for (int i = i0(k / 3 - 1); i < i1(k / 3 - 1) && k != 4; ++i)
        for (int j = j0(k % 3 - 1); j < j1(k % 3 - 1); ++j) n += count(i, j);
    return n;
  }
  // Places in a region with rows `pitch` apart, of the three pixels of packet u of
  // block (i, j) of the tile (dy, dx) away; 16 bits each.
  static __device__ __forceinline__ uint2 places(int i, int j, int u, int dy, int dx, int pitch) {
    unsigned at[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int l = min(3 * u + q, rows(i) * cols(j) - 1), r = l / cols(j);
      at[q] = (K + dy * TH + row0(i) + r) * pitch + K + dx * TW + col0(j) + l - r * cols(j);
    }
    return make_uint2(at[0] | at[1] << 16, at[2]);
  }
};

// Whether a channel's maximum lies beyond tol: the host's comparison
// (GridSolverImpl::beyond), operation by operation.
__device__ __forceinline__ bool res_beyond(const double* maxima, double tol) {
  const volatile double* v = maxima;
  const double a = v[0], b = v[1], c = v[2], m = b < c ? c : b;
  return (a < m ? m : a) > tol;
}

// WHOLE: the region holds the whole grid.  It needs no apron but a lane on
// each side, whose zeros are what a grid's border sees beyond it, and no
// exchange.
template <int R, int W, int LW, int K, bool WHOLE>
__global__ void __launch_bounds__(W * 32, 1) grid_res_kernel(ResArgs A) {
  constexpr int NT = W * 32, NS = NT / LW, H = R * NS, WD = 4 * LW;  // strips, region rows and columns
  __shared__ float4 edge[2][2][NS][LW];
  __shared__ int s_stop;
  __shared__ unsigned s_base, s_nb;
  __shared__ int s_wild, s_done;
  // [H][HP]: the apron (received, or constant) and the tile's ring (to send).
  // Rows K words further apart than their width put a side block's pixels,
  // K a row, into consecutive banks.
  constexpr int HP = WD + K;
  extern __shared__ __align__(16) float halo[];
  // Places in halo[] of the packets to send and to receive, and where the
  // latter lie (-1: no tile that sends).
  using Out = Ring<K, H - 2 * K, WD - 2 * K>;
  constexpr int NP = Out::packets, NI = Out::apron();
  uint2* const t_out = reinterpret_cast<uint2*>(halo + H * HP);
  uint2* const t_in = t_out + NP;
  int* const t_from = reinterpret_cast<int*>(t_in + NI);
  const GridGeom& G = A.G;
  const int lane = threadIdx.x % LW, w = threadIdx.x / LW;  // place in the strip, strip
  constexpr int KL = K / 4;  // apron lanes
  constexpr int TH = H - 2 * K, TW = WD - 2 * K;
  static_assert(H * HP <= 65536 && K % 4 == 0 && K <= kCheck && kCheck % K == 0, "places and periods");
  const int tile = blockIdx.x / 3, c = blockIdx.x - 3 * tile;
  const int ty = tile / A.tiles_x, tx = tile - ty * A.tiles_x;
  constexpr int ap = WHOLE ? 0 : K, al = WHOLE ? 1 : KL;
  constexpr int period = WHOLE ? kCheck : K;  // sweeps between exchanges
  // Tiny values are swept by quarter_sweep in the reference's order rather than
  // by slow_sweep: on an 802x802 grid half of it black 0.975 us a sweep against
  // 1.11 (0.925 without tiny values, 1.00 on the flow kernel), 660x660 0.715
  // against 0.815, 176x1457 0.545 against 0.68.  On the other shapes the second
  // loop cost the first 1-5%, and slow sweeps there are 1-18% slower than it,
  // twice as fast as the launches' all the same.
  constexpr bool ORDERED = W == 8 && K != 8 && !WHOLE;
  const long long org = G.at(ty * TH - ap, tx * TW - 4 * al);  // the region's first pixel
  const long long base = org + (long long)(w * R) * G.pitch + 4 * lane;
  const long long co = c * G.plane;
  if (threadIdx.x == 0) {
    s_stop = 0;
    s_base = *(volatile unsigned*)A.ctl;
  }
  if (threadIdx.x == 0) s_wild = *A.wild != 0;
  if (threadIdx.x == 0) s_done = A.maxima && !res_beyond(A.maxima, A.tol);
  const bool wild = *A.wild != 0;
  float P[R][4], Gq[R][4], L[R][4];
  bool mine = false;  // a masked pixel in the tile interior
  const bool core_lane = lane >= al && lane < LW - al;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const long long p = base + (long long)i * G.pitch;
    const float4 x4 = __ldcg(reinterpret_cast<const float4*>(A.xin + co + p));
    const float4 g4 = ld4(A.g + co + p);
    const uint32_t mk = __ldg(reinterpret_cast<const unsigned*>(A.mask + p));
    const int r = w * R + i;
    mine = mine || (mk != 0 && core_lane && r >= ap && r < H - ap);
    const float x[4] = {x4.x, x4.y, x4.z, x4.w}, gv[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool on = (mk >> (8 * j)) & 0xffu;
      P[i][j] = x[j];
      L[i][j] = on ? __uint_as_float(kMasked) : x[j] == x[j] ? x[j] : __uint_as_float(0x7fc00000u);
      Gq[i][j] = on ? (wild ? gv[j] : __fmul_rn(gv[j], 0.25f)) : __uint_as_float(kNegInf);
    }
    // Apron pixels nobody sends keep these values.
    if (WHOLE) continue;
    if (r < K || r >= H - K || !core_lane) *reinterpret_cast<float4*>(halo + r * HP + 4 * lane) = x4;
  }
  const bool active = __syncthreads_or(mine);
  if (s_done) return;  // in every CTA: nothing was sent, the epochs stay
  const unsigned ebase = s_base;
  // Activity of this and the neighbouring tiles (epoch ebase + 1).
  if (threadIdx.x == 0)
    *(volatile unsigned*)(A.act + blockIdx.x) = ((ebase + 1) << 1) | (active ? 1u : 0u);
  if (threadIdx.x < 32) {
    const int ny = ty + (int)threadIdx.x / 3 - 1, nx = tx + (int)threadIdx.x % 3 - 1;
    bool on = false;
    if (!WHOLE && active && threadIdx.x < 9 && threadIdx.x != 4 && ny >= 0 && nx >= 0 && nx < A.tiles_x &&
        ny * A.tiles_x + nx < A.tiles) {
      const volatile unsigned* q = A.act + 3 * (ny * A.tiles_x + nx) + c;
      unsigned v = *q;
      for (long long spins = 0; (v >> 1) != ((ebase + 1) & 0x7fffffffu); ++spins) {
        if (spins >= A.spin_limit || *(volatile int*)A.error) {
          atomicExch(A.error, 1);
          s_stop = 1;
          break;
        }
        if (spins >= 8) __nanosleep(32);
        v = *q;
      }
      on = v & 1u;
    }
    const unsigned b = __ballot_sync(0xffffffffu, on);
    if (threadIdx.x == 0) s_nb = b;
  }
  __syncthreads();
  if (active && !s_stop) {
    const unsigned nb = s_nb;
    constexpr int NU = (NI + NT - 1) / NT, NO = (NP + NT - 1) / NT;
    constexpr int NB = R < 16 || NU < 6 ? NU : (NU + 1) / 2;  // polled at a time
    if constexpr (!WHOLE) {
#pragma unroll
      for (int i = 0; i < Out::bands; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          for (int u = threadIdx.x; u < Out::count(i, j); u += NT)
            t_out[Out::first(i, j) + u] = Out::places(i, j, u, 0, 0, HP);
      int n = 0;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const int dy = k / 3 - 1, dx = k % 3 - 1;
        if (k == 4) continue;
        // The neighbour at (dy, dx) is read where it faces this tile.
        const int from = (nb >> k) & 1u ? (((int)blockIdx.x + 3 * (dy * A.tiles_x + dx)) * NP) : -1;
#pragma unroll
        for (int i = Out::i0(-dy); i < Out::i1(-dy); ++i)
#pragma unroll
          for (int j = Out::j0(-dx); j < Out::j1(-dx); ++j) {
            for (int u = threadIdx.x; u < Out::count(i, j); u += NT) {
              t_in[n + u] = Out::places(i, j, u, dy, dx, HP);
              t_from[n + u] = from < 0 ? -1 : from + Out::first(i, j) + u;
            }
            n += Out::count(i, j);
          }
      }
    }
    bool slow = wild;
    for (int done = 0; done < A.sweeps; done += period) {
      // The look for tiny values.  What the apron holds next is looked at by
      // its senders, who mark it.
      const auto least = [&] {
        unsigned v = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) v = min(v, tiny_key(P[i][j]));
        return v < tiny_limit(kTiny);
      };
      if (WHOLE || done == 0) {
        slow = __syncthreads_or(least()) || s_wild;
      } else if constexpr (!WHOLE) {
        const int tid = fresh_tid(), ln = tid % LW, st = tid / LW, p = done / K;
        float* const strip = halo + (st * R) * HP + 4 * ln;
        // Send the ring (state after `done` sweeps), through shared memory:
        // from registers it would be R rows of mostly idle stores.
        const bool side_out = ln < 2 * KL || ln >= LW - 2 * KL, side_in = ln < KL || ln >= LW - KL;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int r = st * R + i;
          if (side_out || r < 2 * K || r >= H - 2 * K)
            *reinterpret_cast<float4*>(strip + HP * i) =
                make_float4(P[i][0], P[i][1], P[i][2], P[i][3]);
        }
        if (done % kCheck == 0)
          slow = __syncthreads_or(least()) || s_wild;
        else
          __syncthreads();
        const unsigned want = (s_base + 1 + p) << 1, e = want | (slow ? 1u : 0u);
        uint4* const buf = A.packets + (size_t)((p & 1) * gridDim.x) * NP;
#pragma unroll
        for (int q = 0; q < NO; ++q)
          if ((q + 1) * NT <= NP || tid + q * NT < NP) {
            const uint2 t = t_out[tid + q * NT];
            st_packet(buf + (size_t)blockIdx.x * NP + tid + q * NT, halo[t.x & 0xffffu],
                      halo[t.x >> 16], halo[t.y], e);
          }
        // Receive the neighbours' rings into the apron.
        unsigned marks = 0;
#pragma unroll 1
        for (int q0 = 0; q0 < NU; q0 += NB) {
          const uint2* t = t_in + tid + q0 * NT;
          int from[NB];
          unsigned pend = 0;
#pragma unroll
          for (int q = 0; q < NB; ++q) {
            from[q] = tid + (q0 + q) * NT < NI ? t_from[tid + (q0 + q) * NT] : -1;
            if (from[q] >= 0) pend |= 1u << q;
          }
          for (long long spins = 0; pend; ++spins) {
            ulonglong2 v[NB];
#pragma unroll
            for (int q = 0; q < NB; ++q)
              if ((pend >> q) & 1u) v[q] = ld_packet(buf + from[q]);
#pragma unroll
            for (int q = 0; q < NB; ++q)
              if ((pend >> q) & 1u) {
                const unsigned ev = (unsigned)(v[q].y >> 32);
                if ((ev ^ want) <= 1u) {
                  pend &= ~(1u << q);
                  marks |= ev;
                  const uint2 at = t[q * NT];
                  halo[at.x & 0xffffu] = __uint_as_float((unsigned)v[q].x);
                  halo[at.x >> 16] = __uint_as_float((unsigned)(v[q].x >> 32));
                  halo[at.y] = __uint_as_float((unsigned)v[q].y);
                }
              }
            if (pend && (spins >= A.spin_limit || ((spins & 63) == 63 && *(volatile int*)A.error))) {
              atomicExch(A.error, 1);
              s_stop = 1;
              q0 = NU;
              break;
            }
          }
        }
        slow = __syncthreads_or(marks & 1u) || slow;
        if (s_stop) break;
        // The apron into the strips.
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int r = st * R + i;
          if (side_in || r < K || r >= H - K) {
            const float4 v = *reinterpret_cast<const float4*>(strip + HP * i);
            P[i][0] = v.x;
            P[i][1] = v.y;
            P[i][2] = v.z;
            P[i][3] = v.w;
          }
        }
      }
      const int ks = min(period, A.sweeps - done);
      int s = 0;
      if (!slow && ks >= 2) {
        post_edges<R, NS, LW>(P, 0, lane, w, edge);
        __syncthreads();
#pragma unroll 1
        for (; s + 2 <= ks; s += 2) {
          quarter_sweep<R, NS, LW, false, true>(P, Gq, L, 0, lane, w, edge);
          quarter_sweep<R, NS, LW, false, false>(P, Gq, L, 1, lane, w, edge);
        }
      } else if (ORDERED && !s_wild && ks >= 2) {
        post_edges<R, NS, LW>(P, 0, lane, w, edge);
        __syncthreads();
#pragma unroll 1
        for (; s + 2 <= ks; s += 2) {
          quarter_sweep<R, NS, LW, false, true, false>(P, Gq, L, 0, lane, w, edge);
          quarter_sweep<R, NS, LW, false, false, false>(P, Gq, L, 1, lane, w, edge);
        }
      }
      // An odd last sweep takes this path too (the same values).
#pragma unroll 1
      for (; s < ks; ++s)
        slow_sweep<R, NS, LW>(
            P, Gq, [&](int i, int j) { return __float_as_uint(L[i][j]) == kMasked; },
            s_wild ? 1.f : 4.f, lane, w, edge);
    }
    const int tid = fresh_tid(), ln = tid % LW, st = tid / LW;
    if (ln >= al && ln < LW - al) {
      const int tl = blockIdx.x / 3, tr = tl / A.tiles_x;
      float* const o = A.xout + (int)(blockIdx.x - 3 * tl) * G.plane +
                       G.at(tr * TH - ap + st * R, (tl - tr * A.tiles_x) * TW - 4 * al + 4 * ln);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int r = st * R + i;
        if (r >= ap && r < H - ap)
          *reinterpret_cast<float4*>(o + (long long)i * G.pitch) =
              make_float4(P[i][0], P[i][1], P[i][2], P[i][3]);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_stop) *(volatile int*)A.host_error = 1;
    // Every CTA read the base before it comes here, so the last one may move it.
    __threadfence();
    if (atomicAdd(A.ctl + 1, 1u) == gridDim.x - 1) {
      A.ctl[1] = 0;
      A.ctl[0] = s_base + 2u + (unsigned)((A.sweeps + period - 1) / period);
    }
  }
}

struct ResKernel {
  ResShape shape;
  // Microseconds per sweep measured on the GB300 with many tiles, and with
  // the whole grid in one tile (no exchange).  Neither depends on the grid:
  // every CTA does the same work, whatever their number.
  float many, one;
  int few;  // steps of up to so many sweeps are faster as launches (GridSolverImpl::few_sweeps)
  const void *kernel, *whole;
};

template <int R, int W, int LW, int K>
ResKernel res_make(float many, float one, int few) {
  return {{R, W, 4 * LW, K},
          many,
          one,
          few,
          (const void*)grid_res_kernel<R, W, LW, K, false>,
          (const void*)grid_res_kernel<R, W, LW, 8, true>};
}

// Depth 8 or 16 where a grid fits one region; with many tiles, a deep apron is cheaper than
// more exchanges (8 rows x 64 columns: 0.266 us at 16, 0.345 at 8).  Depth 4
// for the largest tiles, where deeper ones would not fit on the SMs.
const std::vector<ResKernel>& res_kernels() {
  static const std::vector<ResKernel> v = {
      res_make<6, 4, 16, 8>(0.310f, 0.128f, 16),    // tiles of 32 x 48
      res_make<8, 4, 16, 8>(0.345f, 0.161f, 16),    // 48 x 48
      res_make<8, 8, 32, 8>(0.461f, 0.267f, 20),    // 48 x 112
      res_make<6, 4, 16, 16>(0.220f, 0.128f, 16),   // 16 x 32
      res_make<8, 4, 16, 16>(0.266f, 0.161f, 16),   // 32 x 32
      res_make<8, 8, 16, 16>(0.383f, 0.275f, 17),   // 96 x 32
      res_make<8, 8, 32, 16>(0.385f, 0.267f, 17),   // 32 x 96
      res_make<12, 8, 32, 16>(0.523f, 0.376f, 32),  // 64 x 96
      res_make<16, 8, 32, 16>(0.645f, 0.488f, 64),  // 96 x 96
      res_make<16, 8, 32, 4>(0.925f, 0.490f, 17),   // 120 x 120
  };
  return v;
}

const ResKernel* res_kernel(const ResShape& s) {
  for (const ResKernel& k : res_kernels())
    if (k.shape == s) return &k;
  return nullptr;
}

// Packets of a tile, and of its apron (Ring's counts).
int res_ring(const ResShape& s, bool apron) {
  const int h = s.tile_h(), w = s.tile_w(), k = s.depth;
  const auto n = [](int px) { return (px + 2) / 3; };
  const int corner = n(k * k), row = n(k * (w - 2 * k));
  const bool one = h == k;  // a single band of rows
  const int col = one ? 0 : n((h - 2 * k) * k), corners = one ? 2 : 4, sides = one ? 1 : 2;
  if (!apron) return corners * corner + sides * row + 2 * col;
  // North and south, west and east, and the corners.
  return 2 * (2 * corner + row) + 2 * (corners / 2 * corner + col) + 4 * corner;
}

// halo[] and the tables.
size_t res_smem(const ResShape& s) {
  return (size_t)s.region_h() * (s.width + s.depth) * sizeof(float) + res_ring(s, false) * sizeof(uint2) +
         res_ring(s, true) * (sizeof(uint2) + sizeof(int));
}

// SMs of the current device; the kernels' shared-memory limit is raised on
// the first call per device.
int res_sms() {
  static std::atomic<int> cached[64];
  int dev = 0, sms = 0;
  FPIE_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && cached[dev].load(std::memory_order_acquire) > 0)
    return cached[dev].load(std::memory_order_acquire);
  FPIE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  for (const ResKernel& k : res_kernels())
    FPIE_CUDA(cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)res_smem(k.shape)));
  if (dev >= 0 && dev < 64) cached[dev].store(sms, std::memory_order_release);
  return sms;
}

// One where the grid fits a region: its rows, its columns but a lane on each
// side (48x64 with an apron of 8 would be tiles of 32x48; 38x38 then takes
// 0.128 us per sweep instead of 0.161, 64x56 0.160 instead of 0.208).
int res_tiles(const ResShape& s, int n, int m) {
  if (n <= s.region_h() && m <= s.width - 8) return 1;
  return ((n + s.tile_h() - 1) / s.tile_h()) * ((m + s.tile_w() - 1) / s.tile_w());
}

}  // namespace

// A one-region grid needs no exchange before it sweeps.
int res_few(const ResShape& s, int n, int m) {
  const ResKernel* k = res_kernel(s);
  return !k ? 0 : res_tiles(s, n, m) == 1 ? 5 : k->few;
}

static ResShape res_parse(const char* name) {
  ResShape s{0, 0, 0, 0};
  int used = 0;
  if (std::sscanf(name, "p%dw%dx%dk%dr%n", &s.rows, &s.warps, &s.width, &s.depth, &used) != 4 ||
      name[used] != 0 || !res_kernel(s))
    s.rows = 0;
  return s;
}

bool res_is_name(const char* name) { return res_parse(name).rows > 0; }

ResShape res_named(const char* name, int n, int m) {
  ResShape s = res_parse(name);
  if (s.rows && 3LL * res_tiles(s, n, m) > res_sms()) s.rows = 0;
  return s;
}

// The shape with the least measured time whose tiles fit, one (tile, channel)
// per SM.  Measured against the tile kernel the tuner picked before, us per
// sweep: 152x152 0.220 (0.80), 194x194 0.266 (0.71), 251x389 0.385 (0.83),
// 176x1457 0.523 (0.83).  The depth-4 shape runs at 0.92-0.94 at any size,
// the flow kernel according to its 96x96 tiles: with 64 of them or fewer
// (680x680 to 760x760, 600x840) at 0.89-0.96, with more (803x803, 600x1080,
// 240x2400) at 0.95-1.15; so it is taken above 64.
ResShape res_pick(int n, int m) {
  ResShape best{0, 0, 0, 0};
  if ((long long)n * m > (1LL << 21)) return best;  // far more tiles than SMs
  const int sms = res_sms();
  float least = 1e30f;
  for (const ResKernel& k : res_kernels()) {
    const int tiles = res_tiles(k.shape, n, m);
    if (3 * tiles > sms) continue;
    if (k.shape.depth == 4 && ((n + 95) / 96) * ((m + 95) / 96) <= 64) continue;
    const float t = tiles > 1 ? k.many : k.one;
    if (t < least) {
      least = t;
      best = k.shape;
    }
  }
  return best;
}

// The activity words, and two buffers of packets of the shape that needs most.
size_t res_exchange_bytes(const GridGeom& G) {
  size_t most = 0;
  if ((long long)G.n * G.m <= (1LL << 21))
    for (const ResKernel& k : res_kernels()) {
      const int tiles = res_tiles(k.shape, G.n, G.m);
      if (tiles > 1 && 3 * tiles <= res_sms())
        most = std::max(most, (size_t)2 * 3 * tiles * res_ring(k.shape, false) * sizeof(uint4));
    }
  return most + 4096;
}

void launch_res(const GridGeom& G, const ResShape& s, const uint8_t* mask, const float* g,
                const float* xin, float* xout, void* exchange, unsigned* ctl,
                const unsigned* wild, int sweeps, int* error, int* host_error,
                long long spin_limit, cudaStream_t st, const double* maxima, double tol) {
  const ResKernel* k = res_kernel(s);
  FPIE_REQUIRE(k != nullptr, FPIE_ERR_STATE, "no such resident kernel");
  const int tiles = res_tiles(s, G.n, G.m);
  const int tiles_x = tiles == 1 ? 1 : (G.m + s.tile_w() - 1) / s.tile_w();
  FPIE_REQUIRE(3 * tiles <= res_sms() && 3 * tiles <= 1024, FPIE_ERR_STATE,
               "resident kernel: more tiles than SMs");
  // The activity words first: their place does not depend on the shape.
  unsigned* act = static_cast<unsigned*>(exchange);
  uint4* packets = reinterpret_cast<uint4*>(static_cast<char*>(exchange) + 4096);
  ResArgs a{G,    mask,       g,       xin,
            xout, packets,    act,     ctl,
            wild, error,      host_error, std::min(spin_limit, 1LL << 23),
            maxima, tol,      tiles_x, tiles, sweeps};
  void* args[] = {&a};
  FPIE_CUDA(cudaLaunchCooperativeKernel(tiles > 1 ? k->kernel : k->whole, dim3(3 * tiles),
                                        dim3(s.warps * 32), args, tiles > 1 ? res_smem(s) : 0, st));
}

}  // namespace fpie
