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

}  // namespace lat
