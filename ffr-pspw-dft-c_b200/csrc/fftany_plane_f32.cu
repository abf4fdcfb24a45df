// Run-time-length plane kernels, FP32 (complex64) instantiation.
#include "fftany.cuh"

namespace pspw {

template int any_plane<float2, float>(const Basis &, const FastGeo &, cudaStream_t, int,
                                      const float2 *, const float2 *, const float *, float2 *);

}  // namespace pspw
