// Resident grid sweep: one launch per step, one CTA per (tile, channel), all
// co-resident; a tile's state and gradient stay in registers from the first
// sweep to the last, and only the K-pixel ring around it is exchanged with the
// neighbouring tiles, every K sweeps.
//
// What bounds small grids elsewhere is the time between launches or levels
// (a 194x194 grid: 5.6 us per 8-sweep launch, of which ~1.6 us are sweeps):
// launch, region load and store, tail.  Here that is one exchange, and
// regions are cut as small as lets every SM hold one.  Per sweep: 194x194
// 0.298 us (0.71 as launches of 8 sweeps), 251x389 0.407 (0.83), 176x1457
// 0.540 (0.83).
//
// The update is quarter.cuh's.  Each CTA looks for values below 2^-60 every
// 16 sweeps, before an exchange if there is one; one that finds some takes slow
// sweeps until its next look and marks the packets it sends, and a CTA that
// receives a marked packet does the same.
//
// Exchange.  A packet is 8 bytes {value, epoch} in one 64-bit store, two per
// 16-byte access, at the pixel's place in a plane of packets: the reader
// polls the packet itself, so data and readiness arrive together (measured
// one way: 690 cycles, against 1,490 with release and acquire), without a
// fence, a flag or a barrier on the sender's side.  Two buffers alternate.
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
  unsigned long long* packets;  // [2][3][plane]
  unsigned* act;                // [tiles * 3] activity words
  unsigned* ctl;                // [0] epoch base, [1] CTAs that left
  const unsigned* wild;
  int* error;
  long long spin_limit;
  int period;  // sweeps between exchanges (K, or 16 for a single tile)
  int tiles_x, tiles, sweeps;
};

constexpr int kCheck = 16;            // sweeps between range checks
constexpr int kTiny = 60;     // and their limit, 2^-60: exact for 16 sweeps (quarter.cuh)

__device__ __forceinline__ void st_packets(unsigned long long* p, float a, float b, unsigned e) {
  const unsigned long long hi = (unsigned long long)e << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};"
               :
               : "l"(p), "l"(hi | __float_as_uint(a)), "l"(hi | __float_as_uint(b))
               : "memory");
}

__device__ __forceinline__ ulonglong2 ld_packets(const unsigned long long* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
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

// Pixel pairs of a ring `K` wide inside a region of RH x RW pixels starting
// at (r0, r0): whole rows at the top and bottom, K columns on either side of
// the rows between.
template <int K, int RH, int RW>
struct Ring {
  static constexpr int rows = K * RW / 2, side = (RH - 2 * K) * (K / 2);
  static constexpr int pairs = 2 * rows + 2 * side;
  // Row and column (relative to the ring's corner) of pair u.
  static __device__ __forceinline__ void at(int u, int& r, int& c) {
    if (u < 2 * rows) {
      const bool low = u >= rows;
      const int v = low ? u - rows : u;
      r = v / (RW / 2);
      c = 2 * (v - r * (RW / 2));
      if (low) r += RH - K;
    } else {
      int v = u - 2 * rows;
      const bool right = v >= side;
      if (right) v -= side;
      r = K + v / (K / 2);
      c = 2 * (v % (K / 2)) + (right ? RW - K : 0);
    }
  }
};

template <int R, int W, int LW, int K>
__global__ void __launch_bounds__(W * 32, 1) grid_res_kernel(ResArgs A) {
  constexpr int NT = W * 32, NS = NT / LW, H = R * NS, WD = 4 * LW;  // strips, region rows and columns
  __shared__ float4 edge[2][2][NS][LW];
  __shared__ int s_stop;
  __shared__ unsigned s_base, s_nb;
  __shared__ int s_wild;
  // [H][WD]: the apron (received, or constant) and the tile's ring (to send).
  extern __shared__ __align__(16) float halo[];
  // Per pair of pixels to send (then: to receive) its place in a plane of
  // packets and in halo[], relative to the region's first pixel.
  int2* const t_out = reinterpret_cast<int2*>(halo + H * WD);
  int2* const t_in = t_out + Ring<K, H - 2 * K, WD - 2 * K>::pairs;
  // Per thread: its apron pairs that a neighbour sends.
  unsigned* const t_need = reinterpret_cast<unsigned*>(t_in + Ring<K, H, WD>::pairs);
  const GridGeom& G = A.G;
  const int lane = threadIdx.x % LW, w = threadIdx.x / LW;  // place in the strip, strip
  constexpr int KL = K / 4;  // apron lanes
  constexpr int TH = H - 2 * K, TW = WD - 2 * K;
  static_assert(TH >= K && TW >= K && K % 4 == 0 && K <= kCheck && kCheck % K == 0, "rings and aprons");
  const int tile = blockIdx.x / 3, c = blockIdx.x - 3 * tile;
  const int ty = tile / A.tiles_x, tx = tile - ty * A.tiles_x;
  const long long org = G.at(ty * TH - K, tx * TW - K);  // the region's first pixel
  const long long base = org + (long long)(w * R) * G.pitch + 4 * lane;
  const long long co = c * G.plane;
  if (threadIdx.x == 0) {
    s_stop = 0;
    s_base = *(volatile unsigned*)A.ctl;
  }
  if (threadIdx.x == 0) s_wild = *A.wild != 0;
  const bool wild = *A.wild != 0;
  float P[R][4], Gq[R][4], L[R][4];
  bool mine = false;  // a masked pixel in the tile interior
  const bool core_lane = lane >= KL && lane < LW - KL;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const long long p = base + (long long)i * G.pitch;
    const float4 x4 = __ldcg(reinterpret_cast<const float4*>(A.xin + co + p));
    const float4 g4 = ld4(A.g + co + p);
    const uint32_t mk = __ldg(reinterpret_cast<const unsigned*>(A.mask + p));
    const int r = w * R + i;
    mine = mine || (mk != 0 && core_lane && r >= K && r < H - K);
    const float x[4] = {x4.x, x4.y, x4.z, x4.w}, gv[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool on = (mk >> (8 * j)) & 0xffu;
      P[i][j] = x[j];
      L[i][j] = on ? __uint_as_float(kMasked) : x[j] == x[j] ? x[j] : __uint_as_float(0x7fc00000u);
      Gq[i][j] = on ? (wild ? gv[j] : __fmul_rn(gv[j], 0.25f)) : __uint_as_float(kNegInf);
    }
    // Apron pixels nobody sends keep these values.
    if (r < K || r >= H - K || !core_lane) *reinterpret_cast<float4*>(halo + r * WD + 4 * lane) = x4;
  }
  const bool active = __syncthreads_or(mine);
  const unsigned ebase = s_base;
  // Activity of this and the neighbouring tiles (epoch ebase + 1).
  if (threadIdx.x == 0)
    *(volatile unsigned*)(A.act + blockIdx.x) = ((ebase + 1) << 1) | (active ? 1u : 0u);
  if (threadIdx.x < 32) {
    const int ny = ty + (int)threadIdx.x / 3 - 1, nx = tx + (int)threadIdx.x % 3 - 1;
    bool on = false;
    if (active && threadIdx.x < 9 && threadIdx.x != 4 && ny >= 0 && nx >= 0 && nx < A.tiles_x &&
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
    using Out = Ring<K, TH, TW>;  // this tile's outermost K pixels
    using In = Ring<K, H, WD>;   // the apron
    constexpr int NU = (In::pairs + NT - 1) / NT, NO = (Out::pairs + NT - 1) / NT;
    constexpr int NB = R >= 16 ? 4 : NU < 9 ? NU : (NU + 1) / 2;  // polled at a time
    static_assert(NU <= 32, "one bit per pair");
    unsigned need = 0;
    for (int q = 0; q < NU; ++q) {
      const int u = threadIdx.x + q * NT;
      if (u >= In::pairs) break;
      int r, cc;
      In::at(u, r, cc);
      const int k = (r < K ? 0 : r >= H - K ? 6 : 3) + (cc < K ? 0 : cc >= WD - K ? 2 : 1);
      if ((nb >> k) & 1u) need |= 1u << q;
      t_in[u] = make_int2(r * G.pitch + cc, r * WD + cc);
    }
    t_need[threadIdx.x] = need;
    for (int u = threadIdx.x; u < Out::pairs; u += NT) {
      int r, cc;
      Out::at(u, r, cc);
      t_out[u] = make_int2((r + K) * G.pitch + cc + K, (r + K) * WD + cc + K);
    }
    bool slow = wild;
    for (int done = 0; done < A.sweeps; done += A.period) {
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
      if (done == 0 || A.tiles == 1) {
        slow = __syncthreads_or(least()) || s_wild;
      } else {
        const int tid = fresh_tid(), ln = tid % LW, st = tid / LW, p = done / K;
        float* const strip = halo + (st * R) * WD + 4 * ln;
        // Warps that hold rows of the ring or of the apron above or below
        // stage (and reload) their whole strip.
        const bool apron_strip = st * R < K || (st + 1) * R > H - K;
        const bool ring_strip = st * R < 2 * K || (st + 1) * R > H - 2 * K;
        // Send the ring (state after `done` sweeps), through shared memory:
        // from registers it would be R rows of mostly idle stores.
        if (ring_strip || ln < 2 * KL || ln >= LW - 2 * KL) {
#pragma unroll
          for (int i = 0; i < R; ++i)
            *reinterpret_cast<float4*>(strip + WD * i) =
                make_float4(P[i][0], P[i][1], P[i][2], P[i][3]);
        }
        if (done % kCheck == 0)
          slow = __syncthreads_or(least()) || s_wild;
        else
          __syncthreads();
        const unsigned want = (s_base + 1 + p) << 1, e = want | (slow ? 1u : 0u);
        const int tl = blockIdx.x / 3, tr = tl / A.tiles_x;
        unsigned long long* out = A.packets + ((p & 1) * 3 + (int)(blockIdx.x - 3 * tl)) * G.plane +
                                  G.at(tr * TH - K, (tl - tr * A.tiles_x) * TW - K);
#pragma unroll
        for (int q = 0; q < NO; ++q)
          if ((q + 1) * NT <= Out::pairs || tid + q * NT < Out::pairs) {
            const int2 t = t_out[tid + q * NT];
            const float2 v = *reinterpret_cast<const float2*>(halo + t.y);
            st_packets(out + t.x, v.x, v.y, e);
          }
        // Receive the neighbours' rings into the apron.
        unsigned marks = 0;
#pragma unroll 1
        for (int q0 = 0; q0 < NU; q0 += NB) {
          unsigned pend = (t_need[tid] >> q0) & ((1u << NB) - 1u);
          const int2* t = t_in + tid + q0 * NT;
          for (long long spins = 0; pend; ++spins) {
            ulonglong2 v[NB];
#pragma unroll
            for (int q = 0; q < NB; ++q)
              if ((pend >> q) & 1u) v[q] = ld_packets(out + t[q * NT].x);
#pragma unroll
            for (int q = 0; q < NB; ++q)
              if ((pend >> q) & 1u) {
                const unsigned ea = (unsigned)(v[q].x >> 32), eb = (unsigned)(v[q].y >> 32);
                if (((ea ^ want) | (eb ^ want)) <= 1u) {
                  pend &= ~(1u << q);
                  marks |= ea | eb;
                  *reinterpret_cast<float2*>(halo + t[q * NT].y) =
                      make_float2(__uint_as_float((unsigned)v[q].x), __uint_as_float((unsigned)v[q].y));
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
        // The apron into the strips: whole strips at the sides, and in the
        // first and last warps (whose other pixels were staged above).
        if (apron_strip || ln < KL || ln >= LW - KL) {
#pragma unroll
          for (int i = 0; i < R; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(strip + WD * i);
            P[i][0] = v.x;
            P[i][1] = v.y;
            P[i][2] = v.z;
            P[i][3] = v.w;
          }
        }
      }
      const int ks = min(A.period, A.sweeps - done);
      int s = 0;
      if (!slow && ks >= 2) {
        post_edges<R, NS, LW>(P, 0, lane, w, edge);
        __syncthreads();
#pragma unroll 1
        for (; s + 2 <= ks; s += 2) {
          quarter_sweep<R, NS, LW, true>(P, Gq, L, 0, lane, w, edge);
          quarter_sweep<R, NS, LW, false>(P, Gq, L, 1, lane, w, edge);
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
    if (ln >= KL && ln < LW - KL) {
      const int tl = blockIdx.x / 3, tr = tl / A.tiles_x;
      float* const o = A.xout + (int)(blockIdx.x - 3 * tl) * G.plane +
                       G.at(tr * TH - K + st * R, (tl - tr * A.tiles_x) * TW - K + 4 * ln);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int r = st * R + i;
        if (r >= K && r < H - K)
          *reinterpret_cast<float4*>(o + (long long)i * G.pitch) =
              make_float4(P[i][0], P[i][1], P[i][2], P[i][3]);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // Every CTA read the base before it comes here, so the last one may move it.
    __threadfence();
    if (atomicAdd(A.ctl + 1, 1u) == gridDim.x - 1) {
      A.ctl[1] = 0;
      A.ctl[0] = s_base + 2u + (unsigned)((A.sweeps + A.period - 1) / A.period);
    }
  }
}

struct ResKernel {
  ResShape shape;
  // Microseconds per sweep measured on the GB300 with many tiles, and with
  // the whole grid in one tile (no exchange).  Neither depends on the grid:
  // every CTA does the same work, whatever their number.
  float many, one;
  const void* kernel;
};

template <int R, int W, int LW, int K>
ResKernel res_make(float many, float one) {
  return {{R, W, 4 * LW, K}, many, one, (const void*)grid_res_kernel<R, W, LW, K>};
}

// Depth 8 where a grid fits one tile; with many, a deep apron is cheaper than
// more exchanges (8 rows x 64 columns: 0.295 us at 16, 0.367 at 8).
const std::vector<ResKernel>& res_kernels() {
  static const std::vector<ResKernel> v = {
      res_make<6, 4, 16, 8>(0.323f, 0.132f),    // tiles of 32 x 48
      res_make<8, 4, 16, 8>(0.367f, 0.159f),    // 48 x 48
      res_make<8, 8, 32, 8>(0.488f, 0.263f),    // 48 x 112
      res_make<6, 4, 16, 16>(0.249f, 0.207f),   // 16 x 32
      res_make<8, 4, 16, 16>(0.295f, 0.210f),   // 32 x 32
      res_make<8, 8, 16, 16>(0.403f, 0.351f),   // 96 x 32
      res_make<8, 8, 32, 16>(0.404f, 0.260f),   // 32 x 96
      res_make<12, 8, 32, 16>(0.538f, 0.370f),  // 64 x 96
      res_make<16, 8, 32, 16>(0.715f, 0.492f),  // 96 x 96
  };
  return v;
}

const ResKernel* res_kernel(const ResShape& s) {
  for (const ResKernel& k : res_kernels())
    if (k.shape == s) return &k;
  return nullptr;
}

// halo[] and the two tables.
size_t res_smem(const ResShape& s) {
  const size_t h = s.region_h(), w = s.width, k = s.depth;
  const size_t in = w * k + (h - 2 * k) * k, out = (w - 2 * k) * k + (h - 4 * k) * k;
  return h * w * sizeof(float) + (in + out) * sizeof(int2) + s.warps * 32 * sizeof(unsigned);
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

int res_tiles(const ResShape& s, int n, int m) {
  return ((n + s.tile_h() - 1) / s.tile_h()) * ((m + s.tile_w() - 1) / s.tile_w());
}

}  // namespace

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
// sweep: 152x152 0.249 (0.80), 194x194 0.298 (0.71), 251x389 0.407 (0.83),
// 176x1457 0.540 (0.83).
ResShape res_pick(int n, int m) {
  ResShape best{0, 0, 0, 0};
  if ((long long)n * m > (1LL << 21)) return best;  // far more tiles than SMs
  const int sms = res_sms();
  float least = 1e30f;
  for (const ResKernel& k : res_kernels()) {
    const int tiles = res_tiles(k.shape, n, m);
    if (3 * tiles > sms) continue;
    const float t = tiles > 1 ? k.many : k.one;
    if (t < least) {
      least = t;
      best = k.shape;
    }
  }
  return best;
}

// Packets of three channels, two buffers, then an activity word per SM.
size_t res_exchange_bytes(const GridGeom& G) {
  return (size_t)G.plane * 6 * sizeof(unsigned long long) + 4096;
}

void launch_res(const GridGeom& G, const ResShape& s, const uint8_t* mask, const float* g,
                const float* xin, float* xout, void* exchange, unsigned* ctl,
                const unsigned* wild, int sweeps, int* error, long long spin_limit,
                cudaStream_t st) {
  const ResKernel* k = res_kernel(s);
  FPIE_REQUIRE(k != nullptr, FPIE_ERR_STATE, "no such resident kernel");
  const int tiles_x = (G.m + s.tile_w() - 1) / s.tile_w();
  const int tiles = res_tiles(s, G.n, G.m);
  FPIE_REQUIRE(3 * tiles <= res_sms() && 3 * tiles <= 1024, FPIE_ERR_STATE,
               "resident kernel: more tiles than SMs");
  unsigned long long* packets = static_cast<unsigned long long*>(exchange);
  unsigned* act = reinterpret_cast<unsigned*>(packets + 6 * G.plane);
  ResArgs a{G,    mask,       g,       xin,
            xout, packets,    act,     ctl,
            wild, error,      std::min(spin_limit, 1LL << 23),
            tiles > 1 ? s.depth : kCheck, tiles_x, tiles, sweeps};
  void* args[] = {&a};
  FPIE_CUDA(cudaLaunchCooperativeKernel(k->kernel, dim3(3 * tiles), dim3(s.warps * 32), args,
                                        res_smem(s), st));
}

}  // namespace fpie
