// Host driver of the size rules (csrc/sizes.hpp) for test_sizes.py.
#include "../lattice-dev_gb300/csrc/sizes.hpp"

extern "C" long long bin_table(int nx, int ny, int nz) { return lat::bin_table_size(nx, ny, nz); }
