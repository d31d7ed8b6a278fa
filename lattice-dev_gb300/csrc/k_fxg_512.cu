// k_fxg_512.cu -- fixed-point spectral passes over lines padded to 512 points.
#include "k_fxg.cuh"

namespace lat {
int launch_fxg_512(const SepArgs& a, int axis, cudaStream_t s) { return fx::fxg_dispatch<512>(a, axis, s); }
}  // namespace lat
