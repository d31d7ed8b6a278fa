// k_fxg_128.cu -- fixed-point spectral passes over lines padded to 128 points.
#include "k_fxg.cuh"

namespace lat {
int launch_fxg_128(const SepArgs& a, int axis, cudaStream_t s) { return fx::fxg_dispatch<128>(a, axis, s); }
}  // namespace lat
