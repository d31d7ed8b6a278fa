// k_sep_256.cu -- separable spectral passes for lines of 256 points.
#include "k_sep_stream.cuh"

namespace lat {
int launch_sep_256(const SepArgs& a, int axis, cudaStream_t s) {
  // two FP32 fields on a lattice whose passes all form whole tiles (the
  // streamed passes keep zs, not the Laplacian, between passes)
  if (a.stream) return sep::sep_stream_dispatch<256, false>(a, axis, s);
  return sep::sep_dispatch<256>(a, axis, s);
}
int sep_stream_lines_256(int axis) { return sep::stream_lines<256>(axis); }
int sep_columns_256(int nf) { return sep::sep_columns<256>(nf); }
// pairs of one-field runs (ensembles)
int launch_sep_runs_256(const SepArgs& a, int axis, cudaStream_t s) {
  return sep::sep_stream_dispatch<256, true>(a, axis, s);
}
int sep_runs_lines_256(int axis) { return sep::stream_lines<256>(axis); }
}  // namespace lat
