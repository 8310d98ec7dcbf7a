// Device pieces of the Cholesky diagonal blocks and panels: 8 x 8 blocks that
// every lane factors in registers (chol.cu, one CTA per 128 x 128 block;
// batched_chol.cu, one CTA per matrix).
#pragma once
#include "dev_util.cuh"

namespace fb {

namespace {

// The 8 x 8 lower triangle at D (column-major, ld, shared memory, 16-byte
// aligned, ld even) factored by every lane alike: l[i (i + 1) / 2 + k] =
// L(i, k) off the diagonal, ri[k] = 1 / L(k, k).  Returns the first column
// whose pivot is not > 0 (NaN included), -1 if none; what follows it is not
// meaningful then.
__device__ __forceinline__ int chol8_load_factor(const double* D, int ld, double (&l)[36], double (&ri)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int i = k & ~1; i < 8; i += 2) {
      const double2 v = *reinterpret_cast<const double2*>(D + i + k * ld);
      if (i >= k) l[i * (i + 1) / 2 + k] = v.x;
      l[(i + 1) * (i + 2) / 2 + k] = v.y;
    }
  int fail = -1;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double d = l[k * (k + 1) / 2 + k];
    if (!(d > 0.0) && fail < 0) fail = k;
    const double r = rsqrt(d);
    ri[k] = r;
#pragma unroll
    for (int i = k + 1; i < 8; ++i) l[i * (i + 1) / 2 + k] *= r;
#pragma unroll
    for (int c = k + 1; c < 8; ++c)
#pragma unroll
      for (int i = c; i < 8; ++i)
        l[i * (i + 1) / 2 + c] = fma(-l[i * (i + 1) / 2 + k], l[c * (c + 1) / 2 + k], l[i * (i + 1) / 2 + c]);
  }
  return fail;
}

// x := x inv(L)^T for a row x of eight entries (the rows of the block itself
// give its own factor: a pivot's entry d times 1 / sqrt(d)).
__device__ __forceinline__ void chol8_solve(const double (&l)[36], const double (&ri)[8], double (&x)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    x[k] *= ri[k];
#pragma unroll
    for (int c = k + 1; c < 8; ++c) x[c] = fma(-x[k], l[c * (c + 1) / 2 + k], x[c]);
  }
}

}  // namespace

}  // namespace fb
