// Resident grid sweep ("p<R>w<W>x<width>k<K>r"): a whole step in one launch with
// every tile held in registers from its first sweep to its last.
#pragma once

#include <cstddef>
#include <cstdint>

#include "common.cuh"

namespace fpie {

// One shape of the resident kernel: W warps of strips `width` / 4 lanes wide
// and R rows high, an exchange every K sweeps.
struct ResShape {
  int rows, warps, width, depth;
  int region_h() const { return rows * warps * 128 / width; }
  int tile_h() const { return region_h() - 2 * depth; }
  int tile_w() const { return width - 2 * depth; }
  bool operator==(const ResShape& o) const {
    return rows == o.rows && warps == o.warps && width == o.width && depth == o.depth;
  }
};

// The shape with the least predicted time per sweep whose (tile, channel)
// pairs all fit on the device at once; rows == 0 if there is none.
ResShape res_pick(int n, int m);
// The shape named "p<R>w<W>x<width>k<K>r", rows == 0 if there is no such kernel or
// its tiles of an n x m grid do not fit.
ResShape res_named(const char* name, int n, int m);
bool res_is_name(const char* name);
// The sweeps up to which repeated steps of an n x m grid on shape s are faster
// as launches.
int res_few(const ResShape& s, int n, int m);

// Device memory of an exchange over geometry G: two buffers of packets for
// any shape that fits, and the activity words; must be zero before the first
// launch.  ctl: kResCtl words, zero before the
// first launch.
size_t res_exchange_bytes(const GridGeom& G);
constexpr int kResCtl = 4;

// `sweeps` Jacobi sweeps from xin; every tile holding a masked pixel is
// written to xout.  wild: nonzero where the inputs are outside the range in
// which the quartered form is exact (wild in grid.cu).  A wait that exceeds
// spin_limit polls sets *error and *host_error (pinned memory: the host needs no
// copy to know) and the launch stops early.  maxima: the three
// channels' largest residuals of xin, where a launch is queued before the host
// knows them; if none is beyond tol the launch leaves everything as it is.
void launch_res(const GridGeom& G, const ResShape& s, const uint8_t* mask, const float* g,
                const float* xin, float* xout, void* exchange, unsigned* ctl,
                const unsigned* wild, int sweeps, int* error, int* host_error,
                long long spin_limit, cudaStream_t st, const double* maxima = nullptr,
                double tol = 0.0);

}  // namespace fpie
