// k_fxg_64.cu -- fixed-point spectral passes over lines padded to 64 points.
#include "k_fxg.cuh"

namespace lat {
int launch_fxg_64(const SepArgs& a, int axis, cudaStream_t s) { return fx::fxg_dispatch<64>(a, axis, s); }
}  // namespace lat
