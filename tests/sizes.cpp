// Host driver of the size rules (csrc/sizes.hpp) for test_sizes.py.
#include "../lattice-dev_gb300/csrc/sizes.hpp"

extern "C" long long bin_table(int nx, int ny, int nz) { return lat::bin_table_size(nx, ny, nz); }
extern "C" void fd_tile(int nx, int ny, int nz, int fp64, int nsm, int* out) {
  const lat::FdTile t = lat::fd_default_tile(nx, ny, nz, fp64 != 0, nsm);
  out[0] = t.ty;
  out[1] = t.zc;
  out[2] = lat::fd_tile_fits(ny, nz, t.ty, t.zc);
}
