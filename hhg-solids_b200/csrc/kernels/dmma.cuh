// FP64 tensor-core product and 8 x 8 register transpose shared by the propagation kernels.
#pragma once

#include <cuda_runtime.h>

namespace hhg {

// d += A B with mma.m8n8k4.f64 (IEEE double products and sums): lane (g = lane / 4, c = lane % 4) gives
// A[g][c] and B[c][g] and holds D[g][2c], D[g][2c + 1].  Not volatile: the compiler may interleave
// independent accumulations to hide the latency.
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

__device__ __forceinline__ unsigned movmatrix_trans(unsigned x) {
  unsigned r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}
// Transposes an 8 x 8 block of doubles held as (row g, columns 2c, 2c+1) pairs: each of the four
// 16-bit pieces of the two doubles goes through one b16 transpose.
__device__ __forceinline__ void transpose8(double& a, double& b) {
  const unsigned a0 = __double2loint(a), a1 = __double2hiint(a), b0 = __double2loint(b), b1 = __double2hiint(b);
  const unsigned p0 = movmatrix_trans(__byte_perm(a0, b0, 0x5410)), p1 = movmatrix_trans(__byte_perm(a0, b0, 0x7632));
  const unsigned p2 = movmatrix_trans(__byte_perm(a1, b1, 0x5410)), p3 = movmatrix_trans(__byte_perm(a1, b1, 0x7632));
  a = __hiloint2double((int)__byte_perm(p2, p3, 0x5410), (int)__byte_perm(p0, p1, 0x5410));
  b = __hiloint2double((int)__byte_perm(p2, p3, 0x7632), (int)__byte_perm(p0, p1, 0x7632));
}

}  // namespace hhg
