// k_fx_16.cu -- fixed-point spectral passes of FP64 lattices, lines of 16 points.
#include "k_fx.cuh"

namespace lat {
int launch_fx_16(const SepArgs& a, int axis, cudaStream_t s) { return fx::fx_dispatch<16>(a, axis, s); }
}  // namespace lat
