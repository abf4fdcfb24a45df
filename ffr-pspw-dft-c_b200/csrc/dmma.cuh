// The FP64 tensor-core instruction (DMMA), the only tensor-core form of FP64
// arithmetic on sm_100a.
#pragma once

namespace pspw {

// d(16 x 8) += a(16 x 4) b(4 x 8), FP64: lane (g = lane / 4, t = lane % 4)
// holds a = A[g][t], A[g+8][t]; b = B[t][g]; d = D[g][2t], D[g][2t+1],
// D[g+8][2t], D[g+8][2t+1]
__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b));
}

}  // namespace pspw
