// Run-time-length stick kernels, FP64 (complex128) instantiation.
#include "fftany.cuh"

namespace pspw {

template int any_sticks_inv<double2>(const Basis &, const FastGeo &, cudaStream_t, int,
                                     const double2 *, const double2 *, int, int, double2 *);
template int any_sticks_fwd<double2, double>(const Basis &, const FastGeo &, cudaStream_t, int,
                                             const double2 *, const double2 *, const double *,
                                             const double2 *, int, double2 *, int, int,
                                             const RecArg<double2, double> &);

}  // namespace pspw
