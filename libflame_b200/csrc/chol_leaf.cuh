// Device pieces of the Cholesky diagonal blocks and panels: 8 x 8 blocks that
// every lane factors in registers (chol.cu, one CTA per 128 x 128 block), and
// 32 x 32 blocks of a column-major square S (S[r + c * LD], shared memory) that
// one warp factors and publishes column by column while other warps solve rows
// below it one column behind (batched_chol.cu, one CTA per matrix).
#pragma once
#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int CHOL_IB = 32;

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

__device__ __forceinline__ void publish(int* cnt, int v) {
  asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(smem_u32(cnt)), "r"(v) : "memory");
}
__device__ __forceinline__ int published(const int* cnt) {
  int v;
  asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(smem_u32(cnt)) : "memory");
  return v;
}

// One warp factors the w x w diagonal block at (jb, jb).  Every update is
// unconditional (no divergent branches in the chain): a lane only ever reads
// a[c] of its own row for c <= lane, and entries above the diagonal or past
// w never reach those.  After a failing pivot the rest of the block is not
// meaningful; the failing column is what is reported.  Column j goes to S
// (lanes below the diagonal and the pivot), its reciprocal pivot to s_rinv[j],
// then *cnt := base + j + 1.  Columns are published for all of CHOL_IB, so the
// readers' waits always end.
template <int LD>
__device__ __forceinline__ void potrf_diag32(double* S, int jb, int w, int lane, double* s_rinv, int* cnt, int base,
                                             int* s_fail) {
  double a[CHOL_IB];
#pragma unroll
  for (int c = 0; c < CHOL_IB; ++c)  // rows past w: unit pivots
    a[c] = (c <= lane && lane < w) ? S[(jb + lane) + (jb + c) * LD] : (c == lane ? 1.0 : 0.0);
  int fail = -1;
  double d = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
  for (int j = 0; j < CHOL_IB; ++j) {
    if (!(d > 0.0) && fail < 0 && j < w) fail = j;  // <= 0 or NaN
    const double rinv = rsqrt(d), sd = d * rinv;
    a[j] = lane == j ? sd : (lane > j ? a[j] * rinv : a[j]);
    const double lj = a[j];
    double* col = S + jb + (jb + j) * LD;
    if (lane >= j) col[lane] = lj;
    if (lane == 0) s_rinv[j] = rinv;
    if (j + 1 < CHOL_IB) {
      // lane j + 1's next pivot from its own multiplier, then the broadcast
      const double dn = fma(-lj, lj, a[j + 1]);
      d = __shfl_sync(0xffffffffu, dn, j + 1);
    }
    __syncwarp();
    if (lane == 0) publish(cnt, base + j + 1);
#pragma unroll
    for (int c = j + 1; c < CHOL_IB; ++c) a[c] = fma(-lj, col[c], a[c]);
  }
  if (lane == 0 && fail >= 0) *s_fail = jb + fail;
}

// Row r below the diagonal block at (jb, jb), in step with that warp.
// The wait is for another warp of this CTA, which needs nothing from the
// waiting one; it is bounded all the same (*err set when it runs out).
template <int LD>
__device__ __forceinline__ void potrf_row(double* S, int jb, int r, const double* s_rinv, const int* cnt, int base,
                                          int* err) {
  double x[CHOL_IB];
#pragma unroll
  for (int c = 0; c < CHOL_IB; ++c) x[c] = S[r + (jb + c) * LD];
  int seen = base;
#pragma unroll
  for (int j = 0; j < CHOL_IB; ++j) {
    for (int spin = 0; seen < base + j + 1; seen = published(cnt))
      if (++spin > (1 << 20)) {
        atomicExch(err, 61);
        return;
      }
    x[j] *= s_rinv[j];
    S[r + (jb + j) * LD] = x[j];
#pragma unroll
    for (int c = j + 1; c < CHOL_IB; ++c) x[c] = fma(-x[j], S[(jb + c) + (jb + j) * LD], x[c]);
  }
}

}  // namespace

}  // namespace fb
