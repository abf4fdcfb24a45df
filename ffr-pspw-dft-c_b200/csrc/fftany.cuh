// Stick and plane kernels for any grid whose lengths split into two factors
// at run time: the shapes without a compiled kernel of their own
// (fftpath.cuh), i.e. planes with n1 != n2 and lengths such as 22, 38 or 74
// that the reference's grid rule gives (Setup.cpp:20-34).
//
// The data flow, the stick buffer and the permuted orders are those of
// fftpath.cuh; only the factors are run-time values.  A length n = a * b is
// transformed by register DFTs of the block factor a (at most 16) and the
// strided factor b (at most 16, or a prime up to 61).  The kernels switch on
// the factor once per step; every element a thread touches in a step belongs
// to its own work item, so the steps are in place with one barrier between
// them, and one z-plane goes through its whole y-x-V-x-y chain in shared
// memory.  Planes keep full rows [y][x] (odd stride); the y steps walk the
// active columns through an offset table.
//
// What bounds it: shared-memory traffic and issue, as the compiled planes,
// plus the run-time strides (one integer add per element).  The generic
// five-pass path it replaces moved every plane through L2 twice, divided
// integers per element, and took primes as direct sums on a local-memory
// array.  Block H*psi, before -> with these kernels (-> now, with the pair
// projectors too): 50 x 64 x 45, 93 bands FP32 383 -> 124 -> 112 us; 74^3, 32
// bands FP64 10.5 -> 0.58 -> 0.53 ms; six cells of 30..60 points per axis in one
// batch, FP32 2.23 -> 0.72 -> 0.63 ms.  Per point of a plane 6.9 ps (50 x 64,
// FP32) against 4.9 ps of the compiled 64 x 64.
//
// Primes above 13 hold the item's (p - 1) / 2 symmetric pairs in registers
// and loop over the output pairs, with the cosines and sines broadcast from
// a shared-memory table: (p - 1)^2 multiply-adds per transform.  Kernels are
// compiled per class of the largest factor, so small factors do not pay for
// the registers of large primes.  One class holds all primes, 128 threads of 255
// registers in FP64 (the largest primes spill 388 bytes of stores in the plane
// kernel, 228 in the density's; FP32 takes 184 and none): a class of its own for
// p <= 37 at 160 threads and 168 registers spilled more, 727 against 579 us.
#pragma once

#include <algorithm>
#include <type_traits>

#include "fft2.cuh"
#include "fftpath.h"

namespace pspw {
namespace anypath {

// Largest factor of each class.
constexpr int kClassMax[] = {10, 16, 61};
constexpr int kClasses = 3;

inline int class_of(int factor) {
  for (int c = 0; c < kClasses; c++)
    if (factor <= kClassMax[c]) return c;
  return -1;
}

struct AnyAxis {
  int n, a, b;  // n = a * b: block factor, strided factor
  int h;        // (b - 1) / 2 when b is a prime above 16, else 0
};

inline AnyAxis axis_of(const Split &s) { return {s.n, s.a, s.b, s.b > 16 ? (s.b - 1) / 2 : 0}; }

// floor(it / d) for it, d below 2^16 as a multiply-high by ceil(2^32 / d)
inline unsigned magic(int d) { return (unsigned)((0x100000000ull + d - 1) / d); }

// The lines of one step: line l starts at off[l] (when given) or l * ls, its
// elements es apart.
struct AnyLines {
  const int *off;
  int ls, es, nl;
  unsigned mg;  // magic(nl); 0 when nl == 1
  __device__ __forceinline__ void split(int it, int &l, int &j) const {
    j = mg ? (int)__umulhi((unsigned)it, mg) : it;
    l = it - j * nl;
  }
  __device__ __forceinline__ int at(int l) const { return off ? off[l] : l * ls; }
};

enum Kind { kInvStrided, kInvBlock, kMiddle, kFwdBlock, kFwdStrided };

// A strided item with a prime factor P > 13: elements st apart, in place.
// ct[(k-1) * H + (j-1)] = (cos, sin)(2 pi jk / P).
template <int P, int S, bool TW, typename T>
__device__ __forceinline__ void prime_item(T *line, int st, int j0, const T *w, const T *ct) {
  using R = decltype(T::x);
  constexpr int H = (P - 1) / 2;
  T a[H], b[H];
  const T x0 = line[0];
  T s0 = x0;
#pragma unroll
  for (int j = 0; j < H; j++) {
    const T p = line[(1 + j) * st], q = line[(P - 1 - j) * st];
    a[j] = p + q;
    b[j] = p - q;
    s0 = s0 + a[j];
  }
  line[0] = s0;
#pragma unroll 1
  for (int k = 1; k <= H; k++) {
    const T *c = ct + (k - 1) * H;
    // two partial sums each: a shorter chain of dependent multiply-adds
    R mr[2] = {x0.x, 0}, mi[2] = {x0.y, 0}, qr[2] = {0, 0}, qi[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < H; j++) {
      const T t = c[j];
      mr[j & 1] = fma(t.x, a[j].x, mr[j & 1]);
      mi[j & 1] = fma(t.x, a[j].y, mi[j & 1]);
      qr[j & 1] = fma(t.y, b[j].x, qr[j & 1]);
      qi[j & 1] = fma(t.y, b[j].y, qi[j & 1]);
    }
    const T m = mk<T>(mr[0] + mr[1], mi[0] + mi[1]);
    const T q = mul_i<S>(mk<T>(qr[0] + qr[1], qi[0] + qi[1]));
    T u = m + q, v = m - q;
    if (TW && j0) {
      u = cmul(u, twv(w, j0 * k, S));
      v = cmul(v, twv(w, j0 * (P - k), S));
    }
    line[k * st] = u;
    line[(P - k) * st] = v;
  }
}

// One step over all lines with register DFTs of size F (the other factor is
// `fo`).
template <int KIND, int F, typename T, typename R>
__device__ __forceinline__ void step_fixed(T *base, const AnyLines &L, int fo, const T *w,
                                           const T *ct, const R *vplane, int ny) {
  constexpr bool strided = KIND == kInvStrided || KIND == kFwdStrided;
  constexpr int S = (KIND == kFwdBlock || KIND == kFwdStrided) ? -1 : +1;
  constexpr bool TW = KIND == kInvStrided || KIND == kFwdBlock;
  for (int it = threadIdx.x; it < L.nl * fo; it += blockDim.x) {
    int l, j;
    L.split(it, l, j);
    const int st = strided ? fo * L.es : L.es;
    T *line = base + L.at(l) + (strided ? j : j * F) * L.es;
    if constexpr (F > 16) {
      prime_item<F, S, TW>(line, st, j, w, ct);
    } else {
      T v[F];
      R s[KIND == kMiddle ? F : 1];
      if constexpr (KIND == kMiddle) {
#pragma unroll
        for (int i = 0; i < F; i++) s[i] = __ldg(vplane + (size_t)(F * j + i) * ny + l);
      }
#pragma unroll
      for (int i = 0; i < F; i++) v[i] = line[i * st];
      RDft<F, S>::run(v);
      if constexpr (KIND == kMiddle) {
#pragma unroll
        for (int i = 0; i < F; i++) v[i] = mk<T>(s[i] * v[i].x, s[i] * v[i].y);
        RDft<F, -1>::run(v);
      }
      if constexpr (TW || KIND == kMiddle) {
        if (j) {
#pragma unroll
          for (int k = 1; k < F; k++) v[k] = cmul(v[k], twv(w, j * k, TW ? S : -1));
        }
      }
#pragma unroll
      for (int i = 0; i < F; i++) line[i * st] = v[i];
    }
  }
}

// The step of kind KIND along an axis: block steps have register factor a,
// strided steps b.
template <int CLS, int KIND, typename T, typename R>
__device__ __forceinline__ void step(const AnyAxis &x, T *base, const AnyLines &L, const T *w,
                                     const T *ct, const R *vplane, int ny) {
  constexpr bool strided = KIND == kInvStrided || KIND == kFwdStrided;
  const int f = strided ? x.b : x.a, fo = strided ? x.a : x.b;
#define PSPW_F(F)                                                                      \
  case F:                                                                              \
    if constexpr (F <= kClassMax[CLS] && (F <= 16 || strided))                         \
      step_fixed<KIND, F, T, R>(base, L, fo, w, ct, vplane, ny);                       \
    break;
  switch (f) {
    PSPW_F(1) PSPW_F(2) PSPW_F(3) PSPW_F(4) PSPW_F(5) PSPW_F(6) PSPW_F(7) PSPW_F(8)
    PSPW_F(9) PSPW_F(10) PSPW_F(11) PSPW_F(12) PSPW_F(13) PSPW_F(14) PSPW_F(15) PSPW_F(16)
    PSPW_F(17) PSPW_F(19) PSPW_F(23) PSPW_F(29) PSPW_F(31) PSPW_F(37) PSPW_F(41) PSPW_F(43)
    PSPW_F(47) PSPW_F(53) PSPW_F(59) PSPW_F(61)
    default: break;
  }
#undef PSPW_F
}

// n-th roots of unity of an axis and the table of its prime factor
template <typename T>
__device__ __forceinline__ void load_tables(const AnyAxis &x, const T *wg, T *w, T *ct) {
  for (int t = threadIdx.x; t < x.n; t += blockDim.x) w[t] = wg[t];
  for (int t = threadIdx.x; t < x.h * x.h; t += blockDim.x) {
    const int k = t / x.h, j = t - k * x.h;
    ct[t] = wg[((j + 1) * (k + 1)) % x.b * x.a];
  }
}

struct AnyPlane {
  AnyAxis x, y;
  int ls;                    // row stride of the plane (odd)
  unsigned mg_col, mg_row;   // magic of the active columns, of the rows
};

__host__ __device__ inline size_t plane_elems(const AnyPlane &p) {
  return (size_t)p.y.n * p.ls + p.x.n + p.y.n + p.x.h * p.x.h + p.y.h * p.y.h;
}

// shared memory of the plane kernel (the density kernel adds an FP64 plane
// at the next 16-byte boundary)
inline size_t plane_bytes(const AnyPlane &p, int nxa, size_t elem) {
  return elem * plane_elems(p) + sizeof(int) * (size_t)nxa;
}
__host__ __device__ inline size_t up16(size_t n) { return (n + 15) / 16 * 16; }

// Shared-memory views of a plane block.
template <typename T>
struct PlaneMem {
  T *plane, *wx, *wy, *cx, *cy;
  int *xoff;
  __device__ PlaneMem(const AnyPlane &p, unsigned char *raw) {
    plane = reinterpret_cast<T *>(raw);
    wx = plane + p.y.n * p.ls;
    wy = wx + p.x.n;
    cx = wy + p.y.n;
    cy = cx + p.x.h * p.x.h;
    xoff = reinterpret_cast<int *>(cy + p.y.h * p.y.h);
  }
};

template <typename T>
__device__ __forceinline__ void clear_plane(T *plane, int n) {
  // the plane starts on a 16-byte boundary; an odd FP32 element is left over
  const int n16 = (int)((size_t)n * sizeof(T) / 16);
  int4 *p = reinterpret_cast<int4 *>(plane);
  for (int e = threadIdx.x; e < n16; e += blockDim.x) p[e] = make_int4(0, 0, 0, 0);
  if (sizeof(T) == 8 && (n & 1) && threadIdx.x == 0) plane[n - 1] = czero<T>();
}

// One z-plane of one band: y inverse on the active columns, x inverse, times
// V_eff/NNR, x forward, y forward.
template <int CLS, int NT, int MB, typename T, typename R>
__global__ void __launch_bounds__(NT, MB)
    k_plane_any(FastGeo g, AnyPlane p, int n3, const T *__restrict__ wx_g,
                const T *__restrict__ wy_g, const R *__restrict__ vperm, T *__restrict__ S) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PlaneMem<T> m(p, smem_raw);
  const int zp = blockIdx.x, band = blockIdx.y, nx = p.x.n, ny = p.y.n;
  T *Sz = S + ((size_t)band * n3 + zp) * g.ncol;
  clear_plane(m.plane, ny * p.ls);
  load_tables(p.x, wx_g, m.wx, m.cx);
  load_tables(p.y, wy_g, m.wy, m.cy);
  for (int t = threadIdx.x; t < g.nxa; t += blockDim.x) m.xoff[t] = g.xa_list[t];
  __syncthreads();
  for (int c = threadIdx.x; c < g.ncol; c += blockDim.x)
    m.plane[g.col_y[c] * p.ls + g.col_x[c]] = Sz[c];
  __syncthreads();
  const AnyLines cols{m.xoff, 0, p.ls, g.nxa, p.mg_col};
  const AnyLines rows{nullptr, p.ls, 1, ny, p.mg_row};
  const R *vp = vperm + (size_t)zp * ny * nx;
  // one copy of each step kind for both axes
#pragma unroll 1
  for (int s = 0; s < 7; s++) {
    const bool ax = s >= 2 && s <= 4;
    const AnyAxis x = ax ? p.x : p.y;
    const AnyLines L = ax ? rows : cols;
    const T *w = ax ? m.wx : m.wy, *ct = ax ? m.cx : m.cy;
    if (s == 0 || s == 2)
      step<CLS, kInvStrided, T, R>(x, m.plane, L, w, ct, nullptr, 0);
    else if (s == 1)
      step<CLS, kInvBlock, T, R>(x, m.plane, L, w, ct, nullptr, 0);
    else if (s == 3)
      step<CLS, kMiddle, T, R>(x, m.plane, L, w, ct, vp, ny);
    else if (s == 5)
      step<CLS, kFwdBlock, T, R>(x, m.plane, L, w, ct, nullptr, 0);
    else
      step<CLS, kFwdStrided, T, R>(x, m.plane, L, w, ct, nullptr, 0);
    __syncthreads();
  }
  for (int c = threadIdx.x; c < g.ncol; c += blockDim.x)
    Sz[c] = m.plane[g.col_y[c] * p.ls + g.col_x[c]];
}

// Density of a band group on one z-plane (EvalRhoPsi.cpp:139-150): see
// k_plane_rho in fftpath.cuh.
template <int CLS, int NT, typename T>
__global__ void __launch_bounds__(NT, 1)
    k_plane_rho_any(FastGeo g, AnyPlane p, int n3, const T *__restrict__ wx_g,
                    const T *__restrict__ wy_g, const T *__restrict__ S, int nbb,
                    int bands_per_group, const double *__restrict__ wband, size_t acc_off,
                    double *__restrict__ part) {
  using R = decltype(T::x);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const PlaneMem<T> m(p, smem_raw);
  double *acc = reinterpret_cast<double *>(smem_raw + acc_off);
  const int zp = blockIdx.x, grp = blockIdx.y, nx = p.x.n, ny = p.y.n, n12 = nx * ny;
  load_tables(p.x, wx_g, m.wx, m.cx);
  load_tables(p.y, wy_g, m.wy, m.cy);
  for (int t = threadIdx.x; t < g.nxa; t += blockDim.x) m.xoff[t] = g.xa_list[t];
  for (int e = threadIdx.x; e < n12; e += blockDim.x) acc[e] = 0.0;
  const AnyLines cols{m.xoff, 0, p.ls, g.nxa, p.mg_col};
  const AnyLines rows{nullptr, p.ls, 1, ny, p.mg_row};
  const int b0 = grp * bands_per_group, b1 = min(nbb, b0 + bands_per_group);
  for (int band = b0; band < b1; band++) {
    const T *Sz = S + ((size_t)band * n3 + zp) * g.ncol;
    __syncthreads();
    clear_plane(m.plane, ny * p.ls);
    __syncthreads();
    for (int c = threadIdx.x; c < g.ncol; c += blockDim.x)
      m.plane[g.col_y[c] * p.ls + g.col_x[c]] = Sz[c];
    __syncthreads();
#pragma unroll 1
    for (int s = 0; s < 4; s++) {
      const bool ax = s >= 2;
      const AnyAxis x = ax ? p.x : p.y;
      const AnyLines L = ax ? rows : cols;
      const T *w = ax ? m.wx : m.wy, *ct = ax ? m.cx : m.cy;
      if ((s & 1) == 0)
        step<CLS, kInvStrided, T, R>(x, m.plane, L, w, ct, nullptr, 0);
      else
        step<CLS, kInvBlock, T, R>(x, m.plane, L, w, ct, nullptr, 0);
      __syncthreads();
    }
    const double w = wband[band];
    for (int y = threadIdx.x / 32; y < ny; y += blockDim.x / 32)
      for (int x = threadIdx.x & 31; x < nx; x += 32) {
        const T v = m.plane[y * p.ls + x];
        acc[y * nx + x] += w * ((double)v.x * (double)v.x + (double)v.y * (double)v.y);
      }
  }
  __syncthreads();
  double *pp = part + ((size_t)grp * n3 + zp) * n12;
  for (int e = threadIdx.x; e < n12; e += blockDim.x) pp[e] = acc[e];
}

// ---- sticks (k_sticks_inv / k_sticks_fwd of fftpath.cuh)
template <int CLS, int NT, typename T>
__global__ void __launch_bounds__(NT)
    k_sticks_inv_any(FastGeo g, AnyAxis z, int T1, unsigned mg, const T *__restrict__ wz_g,
                     const T *__restrict__ psi, int ld, int ngw_call, T *__restrict__ S) {
  using R = decltype(T::x);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int LS = z.n + 1;
  T *tile = reinterpret_cast<T *>(smem_raw), *wz = tile + T1 * LS, *cz = wz + z.n;
  const int c0 = blockIdx.x * T1, band = blockIdx.y;
  const int nc = min(T1, g.ncol - c0);
  clear_plane(tile, T1 * LS);
  load_tables(z, wz_g, wz, cz);
  __syncthreads();
  const T *pb = psi + (size_t)band * ld;
  const int k0 = g.col_start[c0], k1 = g.col_start[c0 + nc];
  constexpr int U = 4;  // independent gathers in flight per thread
  for (int kb = k0 + threadIdx.x; kb < k1; kb += U * NT) {
    int ig[U], off[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = kb + u * NT;
      ig[u] = k < k1 ? (g.ig_iota ? k : g.sg_ig[k]) : ngw_call;
      off[u] = k < k1 ? g.sg_off[k] : 0;
    }
    T v[U];
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = ig[u] < ngw_call ? pb[ig[u]] : czero<T>();
#pragma unroll
    for (int u = 0; u < U; u++)
      if (ig[u] < ngw_call) tile[off[u]] = v[u];
  }
  __syncthreads();
  const AnyLines L{nullptr, LS, 1, T1, mg};
  step<CLS, kInvStrided, T, R>(z, tile, L, wz, cz, nullptr, 0);
  __syncthreads();
  step<CLS, kInvBlock, T, R>(z, tile, L, wz, cz, nullptr, 0);
  __syncthreads();
  T *Sb = S + (size_t)band * z.n * g.ncol + c0;
  for (int e = threadIdx.x; e < T1 * z.n; e += NT) {
    int t, q;
    L.split(e, t, q);
    if (t < nc) Sb[(size_t)q * g.ncol + t] = tile[t * LS + q];
  }
}

template <int CLS, int NT, typename T, typename R>
__global__ void __launch_bounds__(NT)
    k_sticks_fwd_any(FastGeo g, AnyAxis z, int T1, unsigned mg, const T *__restrict__ wz_g,
                     const T *__restrict__ S, const R *__restrict__ kin,
                     const T *__restrict__ psi, int ld, T *__restrict__ out, int ldo,
                     int ngw_call, RecArg<T, R> rec) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int LS = z.n + 1;
  T *tile = reinterpret_cast<T *>(smem_raw), *wz = tile + T1 * LS, *cz = wz + z.n;
  const int c0 = blockIdx.x * T1, band = blockIdx.y;
  const int nc = min(T1, g.ncol - c0);
  load_tables(z, wz_g, wz, cz);
  const T *Sb = S + (size_t)band * z.n * g.ncol + c0;
  const AnyLines L{nullptr, LS, 1, T1, mg};
  constexpr int U = 4;
  for (int eb = threadIdx.x; eb < T1 * z.n; eb += U * NT) {
    T v[U];
    int o[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int e = eb + u * NT;
      int t, q;
      L.split(e, t, q);
      const bool in = e < T1 * z.n;
      o[u] = in ? t * LS + q : -1;
      v[u] = in && t < nc ? Sb[(size_t)q * g.ncol + t] : czero<T>();
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (o[u] >= 0) tile[o[u]] = v[u];
  }
  __syncthreads();
  step<CLS, kFwdBlock, T, R>(z, tile, L, wz, cz, nullptr, 0);
  __syncthreads();
  step<CLS, kFwdStrided, T, R>(z, tile, L, wz, cz, nullptr, 0);
  __syncthreads();
  const T *pb = psi + (size_t)band * ld;
  T *ob = out + (size_t)band * ldo;
  const T *xb = (rec.on && rec.cg != (R)0) ? rec.xm2 + (size_t)band * rec.ldx : nullptr;
  const int k0 = g.col_start[c0], k1 = g.col_start[c0 + nc];
  for (int kb = k0 + threadIdx.x; kb < k1; kb += U * NT) {
    int ig[U], off[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = kb + u * NT;
      ig[u] = k < k1 ? (g.ig_iota ? k : g.sg_ig[k]) : ngw_call;
      off[u] = k < k1 ? g.sg_off[k] : 0;
    }
    R kk[U];
    T q[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const bool on = ig[u] < ngw_call;
      kk[u] = on ? kin[ig[u]] : (R)0;
      q[u] = on ? pb[ig[u]] : czero<T>();
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (ig[u] < ngw_call) {
        const T f = tile[off[u]];
        T v = mk<T>(kk[u] * q[u].x + f.x, kk[u] * q[u].y + f.y);
        if (rec.on) {
          v = mk<T>(rec.ca * v.x + rec.cb * q[u].x, rec.ca * v.y + rec.cb * q[u].y);
          if (xb) {
            const T x = xb[ig[u]];
            v.x += rec.cg * x.x;
            v.y += rec.cg * x.y;
          }
        }
        ob[ig[u]] = v;
      }
    }
  }
}

// ---- launchers
inline AnyPlane plane_of(const Basis &B) {
  AnyPlane p;
  p.x = axis_of(B.split[0]);
  p.y = axis_of(B.split[1]);
  p.ls = B.n1 | 1;
  p.mg_col = B.nxa > 1 ? magic(B.nxa) : 0;
  p.mg_row = B.n2 > 1 ? magic(B.n2) : 0;
  return p;
}

inline int round32(int n) { return (n + 31) / 32 * 32; }

// Threads of a plane block with a prime factor above 16: one round of the
// strided step's items (lines x block factor), since an item is long, up to
// four warps, which leaves two blocks 255 registers per thread.
constexpr int kPrimeThreads = 128;
inline int prime_threads(const AnyPlane &p, int nxa) {
  int items = 64;
  if (p.x.h) items = std::max(items, p.y.n * p.x.a);
  if (p.y.h) items = std::max(items, nxa * p.y.a);
  return std::min(kPrimeThreads, round32(items));
}

// f(std::integral_constant) of a class, at least `LO`; -1 when there is none
template <int LO, typename F>
int with_class(int cls, F &&f) {
  switch (std::max(cls, cls < 0 ? cls : LO)) {
    case 0: return f(std::integral_constant<int, LO>());
    case 1: return f(std::integral_constant<int, 1>());
    case 2: return f(std::integral_constant<int, 2>());
    default: return -1;
  }
}

inline int plane_class(const AnyPlane &p) {
  return class_of(std::max(std::max(p.x.a, p.x.b), std::max(p.y.a, p.y.b)));
}

}  // namespace anypath

template <typename T, typename R>
int any_plane(const Basis &B, const FastGeo &g, cudaStream_t st, int nbb, const T *wx,
              const T *wy, const R *vperm, T *S) {
  using namespace anypath;
  const AnyPlane p = plane_of(B);
  const size_t sm = plane_bytes(p, g.nxa, sizeof(T));
  const dim3 grid(B.n3, nbb);
  constexpr bool f32 = sizeof(R) == 4;
  return with_class<0>(plane_class(p), [&](auto cls) -> int {
    constexpr int CLS = decltype(cls)::value;
    if constexpr (CLS == 0) {
      if (B.n1 * B.n2 < 6000) {
        // blocks of 256 threads held to the registers of five (FP32: 63 -> 48)
        // or three (FP64: 118 -> 80) per SM; shared memory leaves room for
        // eight and four (six FP32 cells in a batch 683 -> 631 us, 44 bytes of
        // spilled stores included)
        auto k = k_plane_any<CLS, 256, f32 ? 5 : 3, T, R>;
        if (const int rc = smem_allow_max(k)) return rc;
        k<<<grid, 256, sm, st>>>(g, p, B.n3, wx, wy, vperm, S);
        return PSPW_OK;
      }
    }
    constexpr int NT = CLS < 2 ? 512 : kPrimeThreads;
    constexpr int MB = (f32 && CLS == 0) || CLS == 2 ? 2 : 1;
    auto k = k_plane_any<CLS, NT, MB, T, R>;
    if (const int rc = smem_allow_max(k)) return rc;
    // planes of 6000 points or more leave few blocks per SM: 512 threads
    const int nt = CLS >= 2 ? prime_threads(p, g.nxa) : (B.n1 * B.n2 >= 6000 ? 512 : 256);
    k<<<grid, nt, sm, st>>>(g, p, B.n3, wx, wy, vperm, S);
    return PSPW_OK;
  });
}

template <typename T>
int any_plane_rho(const Basis &B, const FastGeo &g, cudaStream_t st, int ngroups, const T *wx,
                  const T *wy, const T *S, int nbb, int bpg, const double *wband, double *part) {
  using namespace anypath;
  const AnyPlane p = plane_of(B);
  const size_t off = up16(plane_bytes(p, g.nxa, sizeof(T)));
  const size_t sm = off + sizeof(double) * (size_t)B.n1 * B.n2;
  return with_class<1>(plane_class(p), [&](auto cls) -> int {
    constexpr int CLS = decltype(cls)::value;
    constexpr int NT = CLS < 2 ? 512 : kPrimeThreads;  // one or two blocks per SM
    auto k = k_plane_rho_any<CLS, NT, T>;
    if (const int rc = smem_allow_max(k)) return rc;
    k<<<dim3(B.n3, ngroups), CLS < 2 ? (B.n1 * B.n2 >= 2048 ? NT : 256) : prime_threads(p, g.nxa),
        sm, st>>>(g, p, B.n3, wx, wy, S, nbb, bpg, wband, off, part);
    return PSPW_OK;
  });
}

template <typename T>
int any_sticks_inv(const Basis &B, const FastGeo &g, cudaStream_t st, int nbb, const T *wz,
                   const T *in, int ld, int ngw, T *S) {
  using namespace anypath;
  const AnyAxis z = axis_of(B.split[2]);
  const int T1 = stick_tile(z.n);
  const size_t sm = sizeof(T) * ((size_t)T1 * (z.n + 1) + z.n + z.h * z.h);
  const dim3 grid((g.ncol + T1 - 1) / T1, nbb);
  return with_class<1>(class_of(std::max(z.a, z.b)), [&](auto cls) -> int {
    constexpr int CLS = decltype(cls)::value;
    constexpr int NT = CLS < 2 ? 256 : 128;
    auto k = k_sticks_inv_any<CLS, NT, T>;
    if (const int rc = smem_allow_max(k)) return rc;
    k<<<grid, NT, sm, st>>>(g, z, T1, T1 > 1 ? magic(T1) : 0, wz, in, ld, ngw, S);
    return PSPW_OK;
  });
}

template <typename T, typename R>
int any_sticks_fwd(const Basis &B, const FastGeo &g, cudaStream_t st, int nbb, const T *wz,
                   const T *S, const R *kin, const T *in, int ld, T *out, int ldo, int ngw,
                   const RecArg<T, R> &ra) {
  using namespace anypath;
  const AnyAxis z = axis_of(B.split[2]);
  const int T1 = stick_tile(z.n);
  const size_t sm = sizeof(T) * ((size_t)T1 * (z.n + 1) + z.n + z.h * z.h);
  const dim3 grid((g.ncol + T1 - 1) / T1, nbb);
  return with_class<1>(class_of(std::max(z.a, z.b)), [&](auto cls) -> int {
    constexpr int CLS = decltype(cls)::value;
    constexpr int NT = CLS < 2 ? 256 : 128;
    auto k = k_sticks_fwd_any<CLS, NT, T, R>;
    if (const int rc = smem_allow_max(k)) return rc;
    k<<<grid, NT, sm, st>>>(g, z, T1, T1 > 1 ? magic(T1) : 0, wz, S, kin, in, ld, out, ldo, ngw,
                            ra);
    return PSPW_OK;
  });
}

}  // namespace pspw
