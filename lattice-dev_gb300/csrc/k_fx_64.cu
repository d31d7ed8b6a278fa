// k_fx_64.cu -- fixed-point spectral passes of FP64 lattices, lines of 64 points.
#include "k_fx.cuh"

namespace lat {
int launch_fx_64(const SepArgs& a, int axis, cudaStream_t s) { return fx::fx_dispatch<64>(a, axis, s); }
}  // namespace lat
