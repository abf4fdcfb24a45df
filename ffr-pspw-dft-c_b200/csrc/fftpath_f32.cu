// Register-FFT local part of H*psi, FP32 (complex64) instantiation, and which
// grids take the register path.
#include <cstdlib>

#include "fftany.cuh"
#include "fftpath.cuh"

namespace pspw {

// The compiled lengths keep their table entry; any other length takes its
// largest prime above 13 as the strided factor, or the factors with the
// smallest maximum.
Split split_for(int n) {
  const NSplit t = nsplit_for(n);
  if (t.n1 > 0) return {n, t.n1, t.n2};
  Split best{n, 0, 0};
  int best_max = 1 << 30;
  auto radix = [](int f) {  // compiled strided factors
    if (f <= 16) return true;
    for (int p : {17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61})
      if (f == p) return true;
    return false;
  };
  for (int b = 1; b <= 61; b++) {
    if (n % b || !radix(b)) continue;
    const int a = n / b;
    if (a > 16) continue;
    const int mx = std::max(a, b);
    // ties: the larger factor as the block factor (contiguous elements)
    if (mx < best_max || (mx == best_max && b <= 16 && a > best.a)) {
      best = {n, a, b};
      best_max = mx;
    }
  }
  return best;
}

void set_fft_paths(Basis *B) {
  const int nr[3] = {B->n1, B->n2, B->n3};
  bool split = !std::getenv("PSPW_GENERIC_FFT");
  for (int i = 0; i < 3; i++) {
    B->split[i] = split_for(nr[i]);
    split = split && B->split[i].a > 0;
  }
  if (!split) return;
  // a block's shared memory: one plane (and for the density its FP64
  // accumulator), or one tile of sticks
  constexpr size_t limit = 227 * 1024;
  const anypath::AnyPlane p = anypath::plane_of(*B);
  const size_t b32 = anypath::plane_bytes(p, B->nxa, sizeof(float2));
  const size_t b64 = anypath::plane_bytes(p, B->nxa, sizeof(double2));
  const anypath::AnyAxis z = anypath::axis_of(B->split[2]);
  const size_t stick =
      sizeof(double2) * ((size_t)stick_tile(z.n) * (z.n + 1) + z.n + z.h * z.h);
  if (stick > limit) return;
  B->fast32 = b32 <= limit;
  B->fast64 = b64 <= limit;
  B->fast_rho = anypath::up16(b64) + sizeof(double) * (size_t)B->n1 * B->n2 <= limit;
}

template int local_fast<float>(pspw_cell *, const FastGeo &, const float2 *, int, float2 *, int,
                               int, int, const ScratchPlan *, const RecArg<float2, float> &);

}  // namespace pspw
