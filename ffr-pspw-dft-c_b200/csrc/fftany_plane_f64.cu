// Run-time-length plane kernels, FP64 (complex128) instantiation.
#include "fftany.cuh"

namespace pspw {

template int any_plane<double2, double>(const Basis &, const FastGeo &, cudaStream_t, int,
                                        const double2 *, const double2 *, const double *,
                                        double2 *);
template int any_plane_rho<double2>(const Basis &, const FastGeo &, cudaStream_t, int,
                                    const double2 *, const double2 *, const double2 *, int, int,
                                    const double *, double *);

}  // namespace pspw
