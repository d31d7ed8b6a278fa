// k_fxg_256.cu -- fixed-point spectral passes over lines padded to 256 points.
#include "k_fxg.cuh"

namespace lat {
int launch_fxg_256(const SepArgs& a, int axis, cudaStream_t s) { return fx::fxg_dispatch<256>(a, axis, s); }
}  // namespace lat
