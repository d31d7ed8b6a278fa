// k_fxr_32.cu -- fixed-point real-to-complex transform, lines of 32 points.
#include "k_fxr.cuh"

namespace lat {
int launch_fxr_rows_32(const void* hi, const void* c, int precision, void* F, int64_t nlines, const void* tw, int nsm,
                       cudaStream_t s) {
  const fx::RowIn in{hi, static_cast<const float*>(c)};
  return fx::fxr_rows_go<32>(in, precision != LAT_FP64, static_cast<double2*>(F), nlines,
                             static_cast<const fx::Tw*>(tw), nsm, s);
}
int launch_fxr_lines_32(void* F, int64_t nlines, int per, int64_t plane, int64_t stride, const void* tw, int nsm,
                        cudaStream_t s) {
  return fx::fxr_lines_go<32>(static_cast<double2*>(F), nlines, per, plane, stride, static_cast<const fx::Tw*>(tw),
                              nsm, s);
}
}  // namespace lat
