// sizes.hpp -- sizes that follow from a lattice's shape, on the host.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace lat {

constexpr int kMaxBins = 2048;  // shells of a spectrum

// Entries of the shell tables by |n|^2 (BinPlan): every |n|^2 of the lattice,
// but none from kMaxBins^2 on, whose modes no spectrum bins.  64-bit: a box
// may be long and thin (131072 x 2 x 2), where (longest side / 2)^2 is beyond 32.
inline int64_t bin_table_size(int nx, int ny, int nz) {
  const int64_t x = nx / 2, y = ny / 2, z = nz / 2;
  return std::min<int64_t>(x * x + y * y + z * z + 1, (int64_t)kMaxBins * kMaxBins);
}

// Rows a block and planes a chunk of the stencil passes before any autotuning:
// 4 rows (8 or 16 where a grid's 65535 blocks along y end first), and the chunk of
// planes with the least estimated time: blocks share the SMs' throughput, so
// the busiest SM's blocks times their planes (one block re-reads and re-sums
// about half a plane in FP64, most of one in FP32), plus the latency of a
// block's own chain where blocks are few.  Against 8 rows and 32 planes for
// every lattice, a leapfrog step: 32^3 7-point FP64 48.4 -> 3.9 us (tuned:
// 3.9), 64^3 48.4 -> 11.9 (10.9), 50 x 40 x 30 GW FP32 47.7 -> 6.1 (6.1), 144 x
// 100 x 90 GW FP64 725 -> 470 (462), 256^3 GW FP32 382 -> 379 (376).
struct FdTile {
  int ty, zc;
};
constexpr int kGridYZ = 65535;  // blocks of a grid along y and along z
inline FdTile fd_default_tile(int nx, int ny, int nz, bool fp64, int nsm) {
  FdTile t{4, 2};
  while (t.ty < 16 && (ny + t.ty - 1) / t.ty > kGridYZ) t.ty *= 2;
  const bool two = !fp64 && nx % 64 == 0;  // two x-sites per thread
  const int64_t cols = (int64_t)((nx + (two ? 63 : 31)) / (two ? 64 : 32)) * ((ny + t.ty - 1) / t.ty);
  const double halo = fp64 ? 0.5 : 0.8;
  const int first = std::max(2, (nz + kGridYZ - 1) / kGridYZ);
  double best = 1e300;
  for (int zc = first; zc <= std::max(first, std::min(64, nz)); ++zc) {
    const int64_t blocks = cols * ((nz + zc - 1) / zc);
    const int64_t busiest = (blocks + nsm - 1) / nsm, rounds = (blocks + 4 * nsm - 1) / (4 * nsm);
    const double cost = busiest * (zc + halo) + 0.35 * rounds * (zc + 3);
    if (cost < best) {
      best = cost;
      t.zc = std::min(zc, nz);
    }
  }
  return t;
}
// whether a stencil pass over these planes can be launched with the tile
inline bool fd_tile_fits(int ny, int nz, int ty, int zc) {
  return (ny + ty - 1) / ty <= kGridYZ && (nz + zc - 1) / zc <= kGridYZ;
}

}  // namespace lat
