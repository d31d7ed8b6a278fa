// k_fx_256.cu -- fixed-point spectral passes of FP64 lattices, lines of 256 points.
#include "k_fx.cuh"

namespace lat {
int launch_fx_256(const SepArgs& a, int axis, cudaStream_t s) { return fx::fx_dispatch<256>(a, axis, s); }
}  // namespace lat
