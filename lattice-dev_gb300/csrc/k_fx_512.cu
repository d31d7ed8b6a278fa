// k_fx_512.cu -- fixed-point spectral passes of FP64 lattices, lines of 512 points.
#include "k_fx.cuh"

namespace lat {
int launch_fx_512(const SepArgs& a, int axis, cudaStream_t s) { return fx::fx_dispatch<512>(a, axis, s); }
}  // namespace lat
