// k_fx_32.cu -- fixed-point spectral passes of FP64 lattices, lines of 32 points.
#include "k_fx.cuh"

namespace lat {
int launch_fx_32(const SepArgs& a, int axis, cudaStream_t s) { return fx::fx_dispatch<32>(a, axis, s); }
}  // namespace lat
