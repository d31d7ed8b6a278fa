// k_fx_128.cu -- fixed-point spectral passes of FP64 lattices, lines of 128 points.
#include "k_fx.cuh"

namespace lat {
int launch_fx_128(const SepArgs& a, int axis, cudaStream_t s) { return fx::fx_dispatch<128>(a, axis, s); }
}  // namespace lat
