// Run-time-length stick kernels, FP32 (complex64) instantiation.
#include "fftany.cuh"

namespace pspw {

template int any_sticks_inv<float2>(const Basis &, const FastGeo &, cudaStream_t, int,
                                    const float2 *, const float2 *, int, int, float2 *);
template int any_sticks_fwd<float2, float>(const Basis &, const FastGeo &, cudaStream_t, int,
                                           const float2 *, const float2 *, const float *,
                                           const float2 *, int, float2 *, int, int,
                                           const RecArg<float2, float> &);

}  // namespace pspw
