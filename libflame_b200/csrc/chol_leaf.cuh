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

constexpr int POTRF_MAX = 128;              // largest block of potrf_block
constexpr int POTRF_LD = POTRF_MAX + 4;     // = 4 mod 16: conflict-free DMMA fragments
constexpr int POTRF_THREADS = 512;

// S(r, c) -= sum_{k < 8} S(r, jb + k) S(c, jb + k) for 8 x 8 tiles: rows and
// columns from lo (a multiple of 8) to b8, tiles on or below the diagonal;
// warp w of nw takes the column tiles w, w + nw, ..., four row tiles at a time
// in flight.  Entries above the diagonal of a diagonal tile are written too:
// nothing reads them.
__device__ __forceinline__ void syrk8_tiles(double* S, int jb, int lo, int b8, int w, int nw, int lane) {
  const int g = lane >> 2, t = lane & 3;
  for (int c = lo + 8 * w; c < b8; c += 8 * nw) {
    const double* pb = S + c + g + (jb + t) * POTRF_LD;
    const double b0 = pb[0], b1 = pb[4 * POTRF_LD];
    for (int r = c; r < b8; r += 32) {
      double a0[4], a1[4], o0[4], o1[4], d0[4], d1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int ru = min(r + 8 * u, b8 - 8);
        const double* pa = S + ru + g + (jb + t) * POTRF_LD;
        const double* o = S + ru + g + (c + 2 * t) * POTRF_LD;
        a0[u] = pa[0];
        a1[u] = pa[4 * POTRF_LD];
        o0[u] = o[0];
        o1[u] = o[POTRF_LD];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        d0[u] = d1[u] = 0.0;
        dmma_884(d0[u], d1[u], a0[u], b0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) dmma_884(d0[u], d1[u], a1[u], b1);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r + 8 * u < b8) {
          double* o = S + r + 8 * u + g + (c + 2 * t) * POTRF_LD;
          o[0] = o0[u] - d0[u];
          o[POTRF_LD] = o1[u] - d1[u];
        }
    }
  }
}

// The b x b (b <= 128) lower triangle in shared memory, S(r, c) at S[r + c *
// POTRF_LD], := its Cholesky factor, by all POTRF_THREADS threads of the CTA.
// Returns the first failing column, -1 if none, in every thread.  s_fail: two
// words of shared memory, -1 (before a barrier); steps take them in turn, since
// a warp may read a step's word while the next step is under way, and every
// warp has to leave in the same step.
__device__ __forceinline__ int potrf_block(double* S, int b, int* s_fail) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b8 = (b + 7) & ~7;
#pragma unroll 1
  for (int jb = 0; jb < b; jb += 8) {
    double x[8];
    int* flag = s_fail + ((jb >> 3) & 1);
    const bool own = warp < 4 && tid >= jb && tid < b8;  // this thread's row takes part
    if (warp < 4) {
      if ((warp << 5) + 31 >= jb) {  // (a) (warps whose rows are all done skip it)
        double l[36], ri[8];
        const int fail = chol8_load_factor(S + jb + jb * POTRF_LD, POTRF_LD, l, ri);
        // the warp that owns the block's rows stores them below: not before
        // the others have read the block
        if (warp == jb >> 5) bar_sync(2, 128 - (jb & ~31));
        else bar_arrive(2, 128 - (jb & ~31));
        if (tid == jb && fail >= 0 && jb + fail < b) *flag = jb + fail;  // rows past b: not pivots
        if (own) {
#pragma unroll
          for (int k = 0; k < 8; ++k) x[k] = S[tid + (jb + k) * POTRF_LD];
          chol8_solve(l, ri, x);
#pragma unroll
          for (int k = 0; k < 8; ++k) S[tid + (jb + k) * POTRF_LD] = x[k];
        }
      }
    } else if (jb > 0 && jb + 8 < b8) {
      syrk8_tiles(S, jb - 8, jb + 8, b8, warp - 4, POTRF_THREADS / 32 - 4, lane);
    }
    __syncthreads();
    if (*flag >= 0) break;
    if (warp < 4) {  // (b)
      if (own && tid >= jb + 8) {
        const double* row = S + jb + 8 + jb * POTRF_LD;  // rows jb + 8 .., this step's columns
        double y[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) y[c] = S[tid + (jb + 8 + c) * POTRF_LD];
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            const double2 v = *reinterpret_cast<const double2*>(row + c + k * POTRF_LD);
            y[c] = fma(-x[k], v.x, y[c]);
            y[c + 1] = fma(-x[k], v.y, y[c + 1]);
          }
#pragma unroll
        for (int c = 0; c < 8; ++c) S[tid + (jb + 8 + c) * POTRF_LD] = y[c];
      }
      bar_sync(1, 128);
    }
  }
  return max(s_fail[0], s_fail[1]);
}

}  // namespace

}  // namespace fb
