// Shared device helpers: complex arithmetic on double2 / float2 and the
// precision traits the kernels are templated on.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace pspw {

template <typename R>
struct Cx;
template <>
struct Cx<double> {
  using T = double2;
};
template <>
struct Cx<float> {
  using T = float2;
};
template <typename R>
using cx = typename Cx<R>::T;

template <typename T>
__host__ __device__ __forceinline__ T mk(decltype(T::x) re, decltype(T::x) im) {
  T r;
  r.x = re;
  r.y = im;
  return r;
}

__host__ __device__ __forceinline__ double2 operator+(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__host__ __device__ __forceinline__ double2 operator-(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__host__ __device__ __forceinline__ double2 operator*(double s, double2 a) {
  return make_double2(s * a.x, s * a.y);
}
// FP32 pairs add in one instruction (add.f32x2, each half rounded as a scalar
// add): the DFT butterflies are mostly complex adds, and every FFT kernel
// issues at 60-75 % of its slots.  FP32 filter of Si64 3.03 -> 2.95 ms.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ unsigned long long f2_bits(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 f2_of(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
#endif
__host__ __device__ __forceinline__ float2 operator+(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_of(r);
#else
  return make_float2(a.x + b.x, a.y + b.y);
#endif
}
__host__ __device__ __forceinline__ float2 operator-(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_of(r);
#else
  return make_float2(a.x - b.x, a.y - b.y);
#endif
}
__host__ __device__ __forceinline__ float2 operator*(float s, float2 a) {
  return make_float2(s * a.x, s * a.y);
}

// a * b
template <typename T>
__device__ __forceinline__ T cmul(T a, T b) {
  return mk<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// conj(a) * b
template <typename T>
__device__ __forceinline__ T cmulc(T a, T b) {
  return mk<T>(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
// acc += a * b
template <typename T>
__device__ __forceinline__ void cfma(T &acc, T a, T b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
}
// acc += conj(a) * b
template <typename T>
__device__ __forceinline__ void cfmac(T &acc, T a, T b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
}

template <typename T>
__device__ __forceinline__ T czero() {
  return mk<T>(0, 0);
}

// complex value converted between precisions
template <typename T, typename S>
__device__ __forceinline__ T ccast(S v) {
  return mk<T>((decltype(T::x))v.x, (decltype(T::x))v.y);
}

}  // namespace pspw
