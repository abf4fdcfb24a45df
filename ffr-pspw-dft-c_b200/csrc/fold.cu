// FP64 Kleinman-Bylander projector products over pairs (+G, -G).
//
// At the Gamma point the sphere holds -G with every G, EIGR(-G) is the
// conjugate of EIGR(G), and a KB form factor is even (s) or odd (p) under
// G -> -G.  With C = f Re E, S = f Im E at +G (f = PKG_A, E = EIGR),
// u = psi(G) + psi(-G) and V = -i (psi(G) - psi(-G)):
//   even p:  beta^H psi =   sum_pairs  C u + S V
//   odd  p:  beta^H psi = i sum_pairs -S u + C V
// and for the back-projection of w (w' = w for even, -i w for odd p)
//   A = sum_p B(u row, p) w'_p,  Q = sum_p B(V row, p) w'_p,
//   out(+G) += A + i Q,          out(-G) += A - i Q,
// with the same real matrix B: rows u hold C (even) or -S (odd), rows V hold
// S or C.  A complex product over the sphere (four real products per pair of
// elements) becomes a real matrix times a complex block over half of it with
// two rows per pair: half the multiply-adds and half the bytes of beta, the
// same sums of the same products in pairs.  The weights fold the i's away:
// w'_p = W_p times the real sums, for both parities.
//
// The symmetry is checked bit for bit for every atom, projector and G when
// the cell is created (any caller's arrays come in); cells without it keep the
// complex GEMM of gemm.cu.  A call over the first ngw G only treats the others
// as absent (psi = 0, nothing written) and stops at the last pair that has one:
// at worst (no G's partner among them) that is the work of the complex GEMM.
//
// Kernels: DMMA tiles as in gemm.cu (warps of 32 x 16 outputs, cp.async
// ring).  A K step of the projection is one group of 8 pairs = 16 real rows:
// the psi values of the pairs land in shared memory as they are, and the
// fragment loads form u and V, so no folded copy of psi exists.  In the
// back-projection the 16 rows of an m16 fragment are the 8 u rows and 8 V
// rows of one group, so a thread holds A and Q of its pairs and writes both
// G's.  What bounds both at many bands: the FP64 tensor pipe, at half the
// complex GEMM's operations.  Si64, 144 bands: 303 + 276 -> 162 + 145 us
// (projection, back-projection; 64 x 48 tiles, DMMA pipe 70 and 62 % busy);
// Si216, 512 bands: the back-projection 4.6 ms, 31 TFLOP/s.  Whole calls: FP64
// filter of Si64 9.51 -> 7.36 ms by these products alone, H*psi of Si216 24.7 ->
// 17.2 ms.  The error of the projections
// against extended precision is unchanged (Si216: 9.0e-15 both ways).  One
// band: matrix-vector kernels, bound by reading B once from L2 or HBM.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "dmma.cuh"
#include "engine.h"
#include "fold.h"
#include "tc.cuh"

namespace pspw {
namespace {

constexpr int kGroup = 8;  // pairs per group; 16 rows of B

// The pair as a call over the first ngw G sees it: -1 for a G that is not
// among them.  (x < y in every pair, so x is missing only where both are.)
__device__ __forceinline__ int2 below(int2 p, int ngw) {
  return make_int2(p.x < ngw ? p.x : -1, p.y < ngw ? p.y : -1);
}

// flags: [0] EIGR symmetric, [1 + 2 (4 s + lm)] even holds, [.. + 1] odd holds
__global__ void k_fold_check(const int2 *__restrict__ pair, int npair, int ngw, int nat, int nsp,
                             const double2 *__restrict__ eigr, const double *__restrict__ pkga,
                             int *flags) {
  const int rows = nat + nsp;
  const long long n = (long long)rows * npair;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / npair), j = (int)(i - (long long)r * npair);
    const int2 p = pair[j];
    const int q = p.y < 0 ? p.x : p.y;  // G = 0 is its own partner
    if (r < nat) {
      const double2 a = eigr[(size_t)r * ngw + p.x], b = eigr[(size_t)r * ngw + q];
      if (!(a.x == b.x && a.y == -b.y)) atomicAnd(&flags[0], 0);
    } else {
      const int s = r - nat;
#pragma unroll
      for (int lm = 0; lm < 4; lm++) {
        const double a = pkga[((size_t)s * ngw + p.x) * 4 + lm];
        const double b = pkga[((size_t)s * ngw + q) * 4 + lm];
        if (!(a == b)) atomicAnd(&flags[1 + 2 * (4 * s + lm)], 0);
        if (!(a == -b)) atomicAnd(&flags[2 + 2 * (4 * s + lm)], 0);
      }
    }
  }
}

// odd[p]: the form factor of projector p is not even
__global__ void k_fold_odd(const int *__restrict__ flags, const int *__restrict__ psp,
                           const int *__restrict__ plm, int nproj,
                           unsigned char *__restrict__ odd) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < nproj) odd[p] = !flags[1 + 2 * (4 * psp[p] + plm[p])];
}

// B: 16 rows per group (8 u rows, then 8 V rows), columns p = blockIdx.y
__global__ void k_fold_build(const int2 *__restrict__ pair, int groups, int ngw,
                             const double2 *__restrict__ eigr, const double *__restrict__ pkga,
                             const int *__restrict__ patom, const int *__restrict__ psp,
                             const int *__restrict__ plm, const unsigned char *__restrict__ odd,
                             double *__restrict__ B) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y;
  if (j >= groups * kGroup) return;
  const int g = pair[j].x;
  double c = 0.0, s = 0.0;
  if (g >= 0) {
    const double2 e = eigr[(size_t)patom[p] * ngw + g];
    const double f = pkga[((size_t)psp[p] * ngw + g) * 4 + plm[p]];
    c = f * e.x;
    s = f * e.y;
  }
  double *b = B + (size_t)p * 16 * groups + (size_t)(j >> 3) * 16 + (j & 7);
  const bool o = odd[p];
  b[0] = o ? -s : c;
  b[8] = o ? c : s;
}

// Tiles of (32 WM) x (16 WN) outputs, warps of 32 x 16; WM 1 or 2, WN 1 to 4.
template <int WM, int WN>
struct Ft {
  // two ring slots for the tiles of four warps: with three, shared memory held
  // 3 of the 4 blocks per SM that registers allow (64 x 32; the 32 x 64 tile
  // measures the same either way, 94.3 and 94.2 us at 128 bands of Si8)
  static constexpr int BM = 32 * WM, BN = 16 * WN, BK = 16, STAGES = WM * WN == 4 ? 2 : 3;
  static constexpr int THREADS = 32 * WM * WN;
  // padded so that the fragment loads of a half warp (8-byte B) or a quarter
  // warp (16-byte psi) hit distinct banks: 4 mod 16 doubles, 4 mod 8 complex
  static constexpr int LDA = BK + 4;    // projection: B as [p][row]
  static constexpr int LDM = BM + 4;    // back-projection: B as [p][row], rows = M
  static constexpr int LDX = BK + 4;    // complex
  static constexpr int P_A = BM * LDA, P_X = BN * LDX;   // doubles, complex per slot
  static constexpr int Q_A = BK * LDM, Q_X = BN * LDX;
  static constexpr size_t P_SLOT = sizeof(double) * P_A + sizeof(double2) * P_X;
  static constexpr size_t Q_SLOT = sizeof(double) * Q_A + sizeof(double2) * Q_X;
  static constexpr size_t P_SMEM = P_SLOT * STAGES, Q_SMEM = Q_SLOT * STAGES;
  static constexpr int MIN_BLOCKS = 16 / (WM * WN) > 8 ? 8 : 16 / (WM * WN);
  // blocks that shared memory lets an SM hold at once
  static constexpr int RESIDENT = (int)(228 * 1024 / (P_SMEM + 1024)) < MIN_BLOCKS
                                      ? (int)(228 * 1024 / (P_SMEM + 1024))
                                      : MIN_BLOCKS;
};

// part or wp over groups [blockIdx.z * gchunk, +gchunk) below `used`: acc(p, b)
template <int WM, int WN>
__global__ void __launch_bounds__(Ft<WM, WN>::THREADS, Ft<WM, WN>::MIN_BLOCKS)
    k_fold_proj(const double *__restrict__ B, const int2 *__restrict__ pair, int groups, int used,
                int ngw, int nproj, const double2 *__restrict__ psi, int ld, int nb, int gchunk,
                const double *__restrict__ w, const unsigned char *__restrict__ odd,
                double2 *__restrict__ wp, double2 *__restrict__ part) {
  using F = Ft<WM, WN>;
  constexpr int BM = F::BM, BN = F::BN, STAGES = F::STAGES, THREADS = F::THREADS;
  extern __shared__ __align__(16) unsigned char raw[];
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int g0 = blockIdx.z * gchunk, g1 = min(used, g0 + gchunk);
  const int nst = g1 - g0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp % WM) * 32, wn = (warp / WM) * 16;
  const int g = lane >> 2, t = lane & 3;
  const size_t rows = 16 * (size_t)groups;
  auto slotA = [&](int s) { return reinterpret_cast<double *>(raw + s * F::P_SLOT); };
  auto slotX = [&](int s) {
    return reinterpret_cast<double2 *>(raw + s * F::P_SLOT + sizeof(double) * F::P_A);
  };
  // thread's psi element of a step: position kk (0-7: +G, 8-15: -G) of band
  // tid / 16 + ...; its pair index is read one step ahead
  const int kk = tid & 15;
  auto index = [&](int st) {
    if (st >= nst) return -1;
    const int2 p = pair[(g0 + st) * kGroup + (kk & 7)];
    const int g = kk < 8 ? p.x : p.y;
    return g < ngw ? g : -1;
  };
  auto load = [&](int st, int slot, int ig) {
    double *As = slotA(slot);
    double2 *Xs = slotX(slot);
    const double *Bg = B + 16 * (size_t)(g0 + st);
#pragma unroll
    for (int e = tid; e < BM * 8; e += THREADS) {  // 16-byte pieces of 16 rows per p
      const int r = e >> 3, c = e & 7;
      const int p = m0 + r;
      const bool ok = p < nproj;
      tc::cp_async16(As + r * F::LDA + 2 * c, Bg + (ok ? (size_t)p * rows : 0) + 2 * c, ok);
    }
#pragma unroll
    for (int e = tid; e < BN * 16; e += THREADS) {
      const int r = e >> 4, b = n0 + r;
      const bool ok = b < nb && ig >= 0;
      tc::cp_async16(Xs + r * F::LDX + kk, ok ? psi + (size_t)b * ld + ig : psi, ok);
    }
  };
  double cr[2][2][4], ci[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) cr[i][j][q] = ci[i][j][q] = 0.0;
#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) {
    if (s < nst) load(s, s, index(s));
    tc::cp_async_commit();
  }
  int ig_next = index(STAGES - 1);
  for (int st = 0; st < nst; st++) {
    tc::cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (st + STAGES - 1 < nst) load(st + STAGES - 1, (st + STAGES - 1) % STAGES, ig_next);
    tc::cp_async_commit();
    ig_next = index(st + STAGES);
    const double *As = slotA(st % STAGES);
    const double2 *Xs = slotX(st % STAGES);
#pragma unroll
    for (int ks = 0; ks < 8; ks += 4) {  // pairs ks .. ks+3: u rows, then V rows
      double au[2][2], av[2][2];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const double *a = As + (wm + i * 16 + g + 8 * h) * F::LDA + ks + t;
          au[i][h] = a[0];
          av[i][h] = a[8];
        }
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const double2 *x = Xs + (wn + j * 8 + g) * F::LDX + ks + t;
        const double2 p = x[0], q = x[8];
        const double ur = p.x + q.x, ui = p.y + q.y;
        const double vr = p.y - q.y, vi = q.x - p.x;  // -i (p - q)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          dmma(cr[i][j], au[i][0], au[i][1], ur);
          dmma(ci[i][j], au[i][0], au[i][1], ui);
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
          dmma(cr[i][j], av[i][0], av[i][1], vr);
          dmma(ci[i][j], av[i][0], av[i][1], vi);
        }
      }
    }
  }
  tc::cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int p = m0 + wm + i * 16 + g + 8 * (q >> 1);
        const int b = n0 + wn + j * 8 + 2 * t + (q & 1);
        if (p >= nproj || b >= nb) continue;
        double2 v = make_double2(cr[i][j][q], ci[i][j][q]);
        if (part) {
          part[((size_t)blockIdx.z * nb + b) * nproj + p] = v;
          continue;
        }
        if (w) v = make_double2(w[p] * v.x, w[p] * v.y);
        else if (odd[p]) v = make_double2(-v.y, v.x);
        wp[(size_t)b * nproj + p] = v;
      }
}

// the K slices in order, then the weight (w) or the plain projection
__global__ void k_fold_reduce(const double2 *__restrict__ part, int nsplit, int nb, int nproj,
                              const double *__restrict__ w, const unsigned char *__restrict__ odd,
                              double2 *__restrict__ wp) {
  const int n = nb * nproj;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double2 s = part[i];
#pragma unroll 8
  for (int k = 1; k < nsplit; k++) s = s + part[(size_t)k * n + i];
  const int p = i % nproj;
  if (w) s = make_double2(w[p] * s.x, w[p] * s.y);
  else if (odd[p]) s = make_double2(-s.y, s.x);
  wp[i] = s;
}

// rows of groups [blockIdx.x * BM / 16, ...) x bands: out(+-G) += alpha (A +- i Q)
template <int WM, int WN>
__global__ void __launch_bounds__(Ft<WM, WN>::THREADS, Ft<WM, WN>::MIN_BLOCKS)
    k_fold_back(const double *__restrict__ B, const int2 *__restrict__ pair, int groups, int used,
                int ngw, int nproj, const double2 *__restrict__ wp, int nb, double2 *out, int ldo,
                double alpha) {
  using F = Ft<WM, WN>;
  constexpr int BM = F::BM, BN = F::BN, BK = F::BK, STAGES = F::STAGES, THREADS = F::THREADS;
  extern __shared__ __align__(16) unsigned char raw[];
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int nst = (nproj + BK - 1) / BK;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp % WM) * 32, wn = (warp / WM) * 16;
  const int g = lane >> 2, t = lane & 3;
  const int rows = 16 * groups;
  auto slotA = [&](int s) { return reinterpret_cast<double *>(raw + s * F::Q_SLOT); };
  auto slotX = [&](int s) {
    return reinterpret_cast<double2 *>(raw + s * F::Q_SLOT + sizeof(double) * F::Q_A);
  };
  auto load = [&](int st, int slot) {
    double *As = slotA(slot);
    double2 *Xs = slotX(slot);
    const int k0 = st * BK;
#pragma unroll
    for (int e = tid; e < BK * (BM / 2); e += THREADS) {  // row pairs of column p
      const int k = e / (BM / 2), c = e % (BM / 2);
      const int p = k0 + k, r = m0 + 2 * c;
      const bool ok = p < nproj && r < rows;
      tc::cp_async16(As + k * F::LDM + 2 * c, ok ? B + (size_t)p * rows + r : B, ok);
    }
#pragma unroll
    for (int e = tid; e < BN * BK; e += THREADS) {
      const int r = e / BK, k = e % BK;
      const int b = n0 + r, p = k0 + k;
      const bool ok = b < nb && p < nproj;
      tc::cp_async16(Xs + r * F::LDX + k, ok ? wp + (size_t)b * nproj + p : wp, ok);
    }
  };
  double cr[2][2][4], ci[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) cr[i][j][q] = ci[i][j][q] = 0.0;
#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) {
    if (s < nst) load(s, s);
    tc::cp_async_commit();
  }
  for (int st = 0; st < nst; st++) {
    tc::cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (st + STAGES - 1 < nst) load(st + STAGES - 1, (st + STAGES - 1) % STAGES);
    tc::cp_async_commit();
    const double *As = slotA(st % STAGES);
    const double2 *Xs = slotX(st % STAGES);
#pragma unroll
    for (int ks = 0; ks < BK; ks += 4) {
      double a[2][2];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) a[i][h] = As[(ks + t) * F::LDM + wm + i * 16 + g + 8 * h];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const double2 v = Xs[(wn + j * 8 + g) * F::LDX + ks + t];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          dmma(cr[i][j], a[i][0], a[i][1], v.x);
          dmma(ci[i][j], a[i][0], a[i][1], v.y);
        }
      }
    }
  }
  tc::cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int grp = (m0 + wm + i * 16) >> 4;
    if (grp >= used) continue;
    const int2 pr = below(pair[grp * kGroup + g], ngw);
    if (pr.x < 0) continue;
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const int b = n0 + wn + j * 8 + 2 * t + c;
        if (b >= nb) continue;
        // fragment rows g and g + 8: A and Q of pair g
        const double ax = cr[i][j][c], ay = ci[i][j][c];
        const double qx = cr[i][j][2 + c], qy = ci[i][j][2 + c];
        double2 *o = out + (size_t)b * ldo;
        const double2 h = o[pr.x];
        o[pr.x] = make_double2(h.x + alpha * (ax - qy), h.y + alpha * (ay + qx));
        if (pr.y >= 0) {
          const double2 l = o[pr.y];
          o[pr.y] = make_double2(l.x + alpha * (ax + qy), l.y + alpha * (ay - qx));
        }
      }
  }
}

// ---- one band
constexpr int kVP = 4;  // projectors per block of the matrix-vector projection

// part[slice][p]: blocks of 4 columns over a slice of the pairs
__global__ void __launch_bounds__(256)
    k_fold_projv(const double *__restrict__ B, const int2 *__restrict__ pair, int groups, int used,
                 int ngw, int nproj, const double2 *__restrict__ psi, int gchunk,
                 const double *__restrict__ w, const unsigned char *__restrict__ odd,
                 double2 *__restrict__ wp, double2 *__restrict__ part) {
  __shared__ double2 red[8][kVP];
  const size_t rows = 16 * (size_t)groups;
  const int p0 = blockIdx.x * kVP;
  const int j0 = blockIdx.y * gchunk * kGroup, j1 = min(used, (blockIdx.y + 1) * gchunk) * kGroup;
  double2 s[kVP];
#pragma unroll
  for (int q = 0; q < kVP; q++) s[q] = make_double2(0.0, 0.0);
#pragma unroll 2
  for (int j = j0 + threadIdx.x; j < j1; j += 256) {
    const int2 pr = below(pair[j], ngw);
    const double2 zero = make_double2(0.0, 0.0);
    const double2 x = pr.x >= 0 ? psi[pr.x] : zero, y = pr.y >= 0 ? psi[pr.y] : zero;
    const double ur = x.x + y.x, ui = x.y + y.y, vr = x.y - y.y, vi = y.x - x.x;
    const double *b = B + (size_t)p0 * rows + (size_t)(j >> 3) * 16 + (j & 7);
#pragma unroll
    for (int q = 0; q < kVP; q++) {
      if (p0 + q >= nproj) break;
      const double c = b[q * rows], d = b[q * rows + 8];
      s[q].x = fma(c, ur, s[q].x);
      s[q].x = fma(d, vr, s[q].x);
      s[q].y = fma(c, ui, s[q].y);
      s[q].y = fma(d, vi, s[q].y);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < kVP; q++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s[q].x += __shfl_down_sync(0xffffffffu, s[q].x, o);
      s[q].y += __shfl_down_sync(0xffffffffu, s[q].y, o);
    }
    if (lane == 0) red[warp][q] = s[q];
  }
  __syncthreads();
  if (threadIdx.x < kVP && p0 + threadIdx.x < nproj) {
    double2 v = red[0][threadIdx.x];
#pragma unroll
    for (int k = 1; k < 8; k++) v = v + red[k][threadIdx.x];
    const int p = p0 + threadIdx.x;
    if (part) {
      part[(size_t)blockIdx.y * nproj + p] = v;
      return;
    }
    if (w) v = make_double2(w[p] * v.x, w[p] * v.y);
    else if (odd[p]) v = make_double2(-v.y, v.x);
    wp[p] = v;
  }
}

// 32 pairs per block, 8 warps over the projectors (p = warp, warp + 8, ...),
// partial sums added in warp order
__global__ void __launch_bounds__(256)
    k_fold_backv(const double *__restrict__ B, const int2 *__restrict__ pair, int groups, int used,
                 int ngw, int nproj, const double2 *__restrict__ wp, double2 *out, double alpha) {
  __shared__ double4 red[8][32];
  const size_t rows = 16 * (size_t)groups;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  const bool on = j < used * kGroup;
  double ax = 0.0, ay = 0.0, qx = 0.0, qy = 0.0;
  if (on) {
    const double *b = B + (size_t)(j >> 3) * 16 + (j & 7);
#pragma unroll 8
    for (int p = warp; p < nproj; p += 8) {
      const double c = b[p * rows], d = b[p * rows + 8];
      const double2 w = wp[p];
      ax = fma(c, w.x, ax);
      ay = fma(c, w.y, ay);
      qx = fma(d, w.x, qx);
      qy = fma(d, w.y, qy);
    }
  }
  red[warp][lane] = make_double4(ax, ay, qx, qy);
  __syncthreads();
  if (warp != 0 || !on) return;
  const int2 pr = below(pair[j], ngw);
  if (pr.x < 0) return;
  const double2 h = out[pr.x], l = pr.y >= 0 ? out[pr.y] : make_double2(0.0, 0.0);
#pragma unroll
  for (int k = 1; k < 8; k++) {
    const double4 r = red[k][lane];
    ax += r.x;
    ay += r.y;
    qx += r.z;
    qy += r.w;
  }
  out[pr.x] = make_double2(h.x + alpha * (ax - qy), h.y + alpha * (ay + qx));
  if (pr.y >= 0) out[pr.y] = make_double2(l.x + alpha * (ax + qy), l.y + alpha * (ay - qx));
}

int sm_count_now() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
  }();
  return n;
}

int ensure_b64(pspw_cell *c) {
  Projectors &P = c->proj;
  Fold &f = P.fold;
  if (f.d_b64) return PSPW_OK;
  const size_t n = 16 * (size_t)f.groups * P.nproj;
  if (cudaMalloc(&f.d_b64, n * sizeof(double)) != cudaSuccess)
    return fail(PSPW_ERR_OOM, "FP64 projector matrix");
  k_fold_build<<<dim3((f.groups * kGroup + 255) / 256, P.nproj), 256, 0, c->stream>>>(
      f.d_pair, f.groups, c->basis.ngw, P.d_eigr64, P.d_pkga64, P.d_patom, P.d_psp, P.d_plm,
      P.d_odd, f.d_b64);
  c->kernel_launches++;
  PSPW_CUDA(cudaGetLastError());
  return PSPW_OK;
}

// Slices of the groups for `tiles` output tiles: what one wave of `target`
// resident blocks holds, or more when a fuller last wave gains 2 % (Si216, 112
// tiles of 64 x 64: two slices fill 76 % of their wave and took 7.8 ms, 13 fill
// 98 % and take 5.9), in slices of four groups or more and at most 96 (the
// partial sums are written and read once more).
int fold_slices(int tiles, int target, int groups) {
  const int most = std::max(1, std::min(96, groups / 4));
  int best = std::max(1, std::min(most, target / tiles));
  double best_fill = std::min(1.0, (double)tiles * best / target);
  for (int n = best + 1; n <= std::min(most, 16); n++) {
    const double waves = (double)tiles * n / target;
    const double fill = waves / std::ceil(waves);
    if (fill > best_fill + 0.02) {
      best = n;
      best_fill = fill;
    }
  }
  return best;
}

template <int WM, int WN>
int launch_proj(pspw_cell *c, const double2 *psi, int ld, int ngw, int nb, double2 *wp,
                const double *w) {
  using F = Ft<WM, WN>;
  const Projectors &P = c->proj;
  const Fold &f = P.fold;
  const int mt = (P.nproj + F::BM - 1) / F::BM, nt = (nb + F::BN - 1) / F::BN;
  const int target = F::RESIDENT * sm_count_now(), used = fold_groups(f, ngw);
  int nsplit = fold_slices(mt * nt, target, used);
  const int gchunk = (used + nsplit - 1) / nsplit;
  nsplit = (used + gchunk - 1) / gchunk;
  double2 *part = nullptr;
  if (nsplit > 1) {
    const int rc = ws_reserve(c, kWsProjPart, sizeof(double2) * (size_t)nsplit * nb * P.nproj,
                              (void **)&part);
    if (rc) return rc;
  }
  auto kern = k_fold_proj<WM, WN>;
  if (const int rc = smem_allow_max(kern)) return rc;
  kern<<<dim3(mt, nt, nsplit), F::THREADS, F::P_SMEM, c->stream>>>(
      f.d_b64, f.d_pair, f.groups, used, ngw, P.nproj, psi, ld, nb, gchunk, w, P.d_odd, wp, part);
  c->kernel_launches++;
  if (nsplit > 1) {
    // small blocks: few outputs with many slices spread over more SMs
    k_fold_reduce<<<(nb * P.nproj + 63) / 64, 64, 0, c->stream>>>(part, nsplit, nb, P.nproj, w,
                                                                 P.d_odd, wp);
    c->kernel_launches++;
  }
  PSPW_CUDA(cudaGetLastError());
  return PSPW_OK;
}

template <int WM, int WN>
int launch_back(pspw_cell *c, const double2 *wp, int ngw, int nb, double2 *out, int ldo,
                double alpha) {
  using F = Ft<WM, WN>;
  const Projectors &P = c->proj;
  const Fold &f = P.fold;
  auto kern = k_fold_back<WM, WN>;
  if (const int rc = smem_allow_max(kern)) return rc;
  const int used = fold_groups(f, ngw);
  const dim3 grid((16 * used + F::BM - 1) / F::BM, (nb + F::BN - 1) / F::BN);
  kern<<<grid, F::THREADS, F::Q_SMEM, c->stream>>>(f.d_b64, f.d_pair, f.groups, used, ngw, P.nproj,
                                                   wp, nb, out, ldo, alpha);
  c->kernel_launches++;
  PSPW_CUDA(cudaGetLastError());
  return PSPW_OK;
}

// The tile width that pads the bands least (ties to the wider, which re-reads
// B less): 64, 48 or 32 bands, 16 for at most 16.
int tile_bands(int nb) {
  if (nb <= 16) return 16;
  int best = 64, pad = (nb + 63) / 64 * 64;
  for (int w : {48, 32})
    if ((nb + w - 1) / w * w < pad) {
      best = w;
      pad = (nb + w - 1) / w * w;
    }
  return best;
}

}  // namespace

int fold_prepare(pspw_cell *c, const std::vector<int> &col_x, const std::vector<int> &col_y,
                 const std::vector<int> &col_of_xy, const std::vector<int> &col_start,
                 const std::vector<int> &sg_z, const std::vector<int> &order) {
  const Basis &B = c->basis;
  Projectors &P = c->proj;
  if (P.nproj <= 0) return PSPW_OK;
  const int ngw = B.ngw;
  // The partner of G sits at the negated grid index: in the stick (-x, -y), whose
  // z's are the negated ones of G's stick in reverse, after z = 0.  partner[k]:
  // stick-list position of the partner of position k.
  std::vector<int> partner(ngw);
  for (int k = 0; k < B.ncol; k++) {
    const int x = col_x[k], y = col_y[k], k0 = col_start[k], m = col_start[k + 1] - k0;
    const int q = col_of_xy[(x ? B.n1 - x : 0) + (size_t)B.n1 * (y ? B.n2 - y : 0)];
    if (q < 0 || col_start[q + 1] - col_start[q] != m) return PSPW_OK;
    const int zero = sg_z[k0] == 0;
    for (int i = 0; i < m; i++) {
      const int z = sg_z[k0 + i], j = col_start[q] + (i < zero ? 0 : m - 1 - i + zero);
      if (i > 0 && z == sg_z[k0 + i - 1]) return PSPW_OK;  // two G on one grid point
      if (sg_z[j] != (z ? B.n3 - z : 0)) return PSPW_OK;
      partner[k0 + i] = j;
    }
  }
  int npair = 0;
  for (int k = 0; k < ngw; k++) npair += partner[k] >= k;
  const int groups = (npair + kGroup - 1) / kGroup;
  // one allocation and one copy: the pair tables of both orders, the check's
  // flags, and the odd marks (device only)
  const size_t np = (size_t)groups * kGroup, nflags = 1 + 8 * (size_t)P.nsp;
  std::vector<int2> host(2 * np + (nflags + 1) / 2, make_int2(-1, -1));
  int2 *nat = host.data(), *stick = nat + np;
  int *flags = reinterpret_cast<int *>(stick + np);
  std::fill(flags, flags + nflags, 1);
  std::vector<int> nat_partner(ngw);
  for (int k = 0; k < ngw; k++) {
    const int q = partner[k];
    nat_partner[order[k]] = order[q];
    if (q >= k) *stick++ = make_int2(k, q == k ? -1 : q);
  }
  for (int g = 0; g < ngw; g++)
    if (nat_partner[g] >= g) *nat++ = make_int2(g, nat_partner[g] == g ? -1 : nat_partner[g]);
  Fold &f = P.fold, &fs = c->stick.fold;
  f.groups = fs.groups = groups;
  for (int g = 0; g < groups; g++) {  // (the last group has a pair too)
    f.first.push_back(host[(size_t)g * kGroup].x);
    fs.first.push_back(host[np + (size_t)g * kGroup].x);
  }
  if (cudaMalloc(&P.fold_mem, sizeof(int2) * host.size() + P.nproj) != cudaSuccess)
    return fail(PSPW_ERR_OOM, "G pairs");
  f.d_pair = static_cast<int2 *>(P.fold_mem);
  fs.d_pair = f.d_pair + np;
  int *d_flags = reinterpret_cast<int *>(fs.d_pair + np);
  P.d_odd = reinterpret_cast<unsigned char *>(f.d_pair + host.size());
  cudaStream_t st = c->stream;
  PSPW_CUDA(cudaMemcpyAsync(P.fold_mem, host.data(), sizeof(int2) * host.size(),
                            cudaMemcpyHostToDevice, st));
  const long long n = (long long)(P.nat + P.nsp) * npair;
  k_fold_check<<<(unsigned)std::min<long long>((n + 255) / 256, 148 * 16), 256, 0, st>>>(
      f.d_pair, npair, ngw, P.nat, P.nsp, P.d_eigr64, P.d_pkga64, d_flags);
  k_fold_odd<<<(P.nproj + 255) / 256, 256, 0, st>>>(d_flags, P.d_psp, P.d_plm, P.nproj, P.d_odd);
  c->kernel_launches += 2;
  PSPW_CUDA(cudaGetLastError());
  PSPW_CUDA(cudaMemcpyAsync(flags, d_flags, nflags * sizeof(int), cudaMemcpyDeviceToHost, st));
  PSPW_CUDA(cudaStreamSynchronize(st));
  bool ok = flags[0] != 0;
  for (int s = 0; s < P.nsp && ok; s++)
    for (int lm = 0; lm < P.sp_lm[s]; lm++)
      if (P.sp_na[s] > 0)
        ok = ok && (flags[1 + 2 * (4 * s + lm)] || flags[2 + 2 * (4 * s + lm)]);
  P.sp_odd.assign(P.nsp, 0u);
  for (int s = 0; s < P.nsp; s++)
    for (int lm = 0; lm < 4; lm++)
      if (!flags[1 + 2 * (4 * s + lm)]) P.sp_odd[s] |= 1u << lm;
  f.ok = fs.ok = ok;
  return PSPW_OK;
}

int fold_groups(const Fold &f, int ngw) {
  return (int)(std::lower_bound(f.first.begin(), f.first.end(), ngw) - f.first.begin());
}

int fold_project64(pspw_cell *c, const double2 *psi, int ld, int ngw, int nb, double2 *wp,
                   bool plain) {
  int rc = ensure_b64(c);
  if (rc) return rc;
  const Projectors &P = c->proj;
  const Fold &f = P.fold;
  const double *w = plain ? nullptr : P.d_pw64;
  if (nb == 1) {
    // slices of 64 groups (two rounds of 256 threads) or more, four blocks per
    // SM; up to 512 groups (a sphere of 8192 G) one slice, which needs no
    // reduction launch.  Calls of 256 projectors, one slice against several:
    // 379 groups 30.8 / 35.6 us, 584 33.8 / 37.1, 696 35.8 / 34.4, 1490 58.6 /
    // 53.2; of 32 projectors, 369 groups 22.5 / 23.6
    const int pt = (P.nproj + kVP - 1) / kVP;
    const int used = fold_groups(f, ngw);
    int nsplit = used <= 512 ? 1
                             : std::max(1, std::min((used + 63) / 64, 4 * sm_count_now() / pt));
    const int gchunk = (used + nsplit - 1) / nsplit;
    nsplit = (used + gchunk - 1) / gchunk;
    double2 *part = nullptr;
    if (nsplit > 1) {
      rc = ws_reserve(c, kWsProjPart, sizeof(double2) * (size_t)nsplit * P.nproj, (void **)&part);
      if (rc) return rc;
    }
    k_fold_projv<<<dim3(pt, nsplit), 256, 0, c->stream>>>(f.d_b64, f.d_pair, f.groups, used, ngw,
                                                          P.nproj, psi, gchunk, w, P.d_odd, wp,
                                                          part);
    c->kernel_launches++;
    if (nsplit > 1) {
      k_fold_reduce<<<(P.nproj + 127) / 128, 128, 0, c->stream>>>(part, nsplit, 1, P.nproj, w,
                                                                  P.d_odd, wp);
      c->kernel_launches++;
    }
    PSPW_CUDA(cudaGetLastError());
    return PSPW_OK;
  }
  // 32-row tiles where 64-row ones would pad the projectors by more than a
  // tenth (32 projectors: half the tile)
  const int r64 = (P.nproj + 63) / 64 * 64, r32 = (P.nproj + 31) / 32 * 32;
  const bool narrow = 10 * r64 > 11 * r32;
  switch (tile_bands(nb)) {
    case 64:
      return narrow ? launch_proj<1, 4>(c, psi, ld, ngw, nb, wp, w)
                    : launch_proj<2, 4>(c, psi, ld, ngw, nb, wp, w);
    case 48:
      return narrow ? launch_proj<1, 3>(c, psi, ld, ngw, nb, wp, w)
                    : launch_proj<2, 3>(c, psi, ld, ngw, nb, wp, w);
    case 32:
      return narrow ? launch_proj<1, 2>(c, psi, ld, ngw, nb, wp, w)
                    : launch_proj<2, 2>(c, psi, ld, ngw, nb, wp, w);
    default:
      return narrow ? launch_proj<1, 1>(c, psi, ld, ngw, nb, wp, w)
                    : launch_proj<2, 1>(c, psi, ld, ngw, nb, wp, w);
  }
}

int fold_backproject64(pspw_cell *c, const double2 *wp, int ngw, int nb, double2 *out, int ldo,
                       double alpha) {
  const Projectors &P = c->proj;
  const Fold &f = P.fold;
  const int used = fold_groups(f, ngw);
  if (nb == 1) {
    k_fold_backv<<<(used * kGroup + 31) / 32, 256, 0, c->stream>>>(
        f.d_b64, f.d_pair, f.groups, used, ngw, P.nproj, wp, out, alpha);
    c->kernel_launches++;
    PSPW_CUDA(cudaGetLastError());
    return PSPW_OK;
  }
  // 32-row tiles (two groups) where 64-row ones would leave SMs without a block
  const int bands = tile_bands(nb);
  const bool few = (used + 3) / 4 * ((nb + bands - 1) / bands) < sm_count_now();
  switch (bands) {
    case 64:
      return few ? launch_back<1, 4>(c, wp, ngw, nb, out, ldo, alpha)
                 : launch_back<2, 4>(c, wp, ngw, nb, out, ldo, alpha);
    case 48:
      return few ? launch_back<1, 3>(c, wp, ngw, nb, out, ldo, alpha)
                 : launch_back<2, 3>(c, wp, ngw, nb, out, ldo, alpha);
    case 32:
      return few ? launch_back<1, 2>(c, wp, ngw, nb, out, ldo, alpha)
                 : launch_back<2, 2>(c, wp, ngw, nb, out, ldo, alpha);
    default:
      return few ? launch_back<1, 1>(c, wp, ngw, nb, out, ldo, alpha)
                 : launch_back<2, 1>(c, wp, ngw, nb, out, ldo, alpha);
  }
}

}  // namespace pspw
