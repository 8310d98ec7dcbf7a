// Batched FP64 Cholesky (+ solves, log-determinants) for many small matrices
// of uneven sizes, orders up to 512: one CTA per matrix, matrices from an
// atomic counter in a host-chosen order (largest first).
//
// Semantics of FLA_Chol per matrix (src/lapack/dec/chol/front/flamec/
// FLA_Chol.c:16-29): lower triangle only, stopping at the first pivot that is
// not > 0 (NaN included), its zero-based column reported; a matrix that fails
// holds L in the columns before it (of the failing panel, the diagonal block's
// rows), the failing pivot at its place, and keeps its right-hand sides.
//
// Right-looking in panels of 32 columns, in place (148 resident triangles of
// order 512 are 155 MB, past the L2: they move 1.3 GB through HBM, 0.3 GB in and
// out would do, and 68 % of the accesses hit L2):
//   panel   the block column in shared memory, eight columns a step: one warp
//           factors the 8 x 8 block in registers and solves the diagonal
//           block's rows, the other warps the rows below beside its next step;
//   update  A22 -= L21 L21^T (lower) on the FP64 tensor cores, 16 x 32 warp
//           tiles, both operands from the panel in shared memory.
// The right-hand sides are rows below the matrix (kept in shared memory), so
// the forward substitution comes with the factorization; the backward one
// takes L(below, block)^T x on the tensor cores, block by block.  Bound by the
// update's tiles for the large orders (148 matrices of order 512: 38.7 of 65
// thousand cycles a panel, the FP64 tensor pipe at 34 % and the L1 data path at
// 66 % of their rates over the whole kernel), by the panels' pivot chain (11.7
// thousand there) for the small ones.  Orders up to 256 run in CTAs of 256 threads, two per
// SM, so that one matrix's chain overlaps the other's updates; 257 to 512 in
// CTAs of 512.
// Measured: 2500 matrices, n uniform in 8..512, 4 right-hand sides: 11.9 ms
// left-looking with one CTA of 512 threads per SM (chol_batched_dmma_kernel,
// which keeps the orders above 512); 4.5 ms right-looking with panels factored
// column by column and a row per thread in the backward substitution; 3.9 ms
// in this form.
#include <algorithm>

#include "batched.h"
#include "chol_leaf.cuh"
#include "common.h"

namespace fb {

namespace {

constexpr int CW_ = 32;           // panel width
constexpr int CRHS = 8;           // right-hand sides

template <int NT>
struct ChB {
  static constexpr int NW = NT / 32;
  static constexpr int LD = NT + 20;        // rows of the panel: NT, the right-hand sides, a tile's rest; = 4 mod 16
  static constexpr int LDR = NT;            // right-hand side q at sR[q * LDR]
  static constexpr size_t SMEM = sizeof(double) * ((size_t)LD * CW_ + (size_t)CRHS * LDR + CW_);
  static constexpr int MINB = NT == 256 ? 2 : 1;
};

// Entries s .. s + 7 of row r of the panel less the products of its columns
// before s with the diagonal block's rows.
template <int LD>
__device__ __forceinline__ void row_minus(const double* P, int r, int s, double (&x)[8]) {
#pragma unroll
  for (int c = 0; c < 8; ++c) x[c] = P[r + (s + c) * LD];
#pragma unroll 4
  for (int k = 0; k < s; ++k) {
    const double v = P[r + k * LD];
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 b = *reinterpret_cast<const double2*>(P + s + c + k * LD);
      x[c] = fma(-v, b.x, x[c]);
      x[c + 1] = fma(-v, b.y, x[c + 1]);
    }
  }
}

// x := x inv(L)^T for the factored 8 x 8 block at column s, its reciprocal
// pivots in rinv.
template <int LD>
__device__ __forceinline__ void row_solve(const double* P, int s, const double* rinv, double (&x)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    x[k] *= rinv[s + k];
    const double* col = P + s + (s + k) * LD;
#pragma unroll
    for (int c = k + 1; c < 8; ++c) x[c] = fma(-x[k], col[c], x[c]);
  }
}

template <int LD>
__device__ __forceinline__ void store8(double* P, int r, int s, const double (&x)[8]) {
#pragma unroll
  for (int c = 0; c < 8; ++c) P[r + (s + c) * LD] = x[c];
}

template <int NT>
__global__ void __launch_bounds__(NT, ChB<NT>::MINB) chol_batched_f64_kernel(BatchArgs<double> a) {
  using B = ChB<NT>;
  constexpr int NW = B::NW, LD = B::LD, LDR = B::LDR;
  extern __shared__ __align__(16) double chb_sm[];
  double* P = chb_sm;                      // panel: row r (from the panel's first), column c at P[r + c * LD]
  double* sR = P + (size_t)LD * CW_;       // right-hand sides
  double* rinv = sR + CRHS * LDR;          // [32] the panel's reciprocal pivots
  __shared__ int s_next, s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_next = atomicAdd(a.counter, 1);
      s_fail = -1;
    }
    __syncthreads();
    if (s_next >= a.count) break;
    const int mi = a.order[s_next];
    const int n = a.n[mi], nrhs = a.B ? a.nrhs : 0;
    const long ld = a.ld[mi];
    double* G = a.A[mi];
    for (int e = tid; e < n * nrhs; e += NT) {
      const int r = e % n, q = e / n;
      cp_async8(sR + r + q * LDR, a.B[mi] + (long)r + (long)q * a.ldb[mi]);
    }
    int fail = -1;  // the same in every thread
    for (int j = 0; j < n; j += CW_) {
      const int w = min(CW_, n - j), R = n - j;
      const int RB = max(R, CW_);  // panel rows RB ..: the right-hand sides (past the whole diagonal block)
      for (int c = warp; c < w; c += NW)
        for (int r = c + lane; r < R; r += 32) cp_async8(P + r + c * LD, G + (long)(j + r) + (long)(j + c) * ld);
      if (w < CW_)  // the last panel: unit pivots past the matrix
        for (int e = tid; e < CW_ * CW_; e += NT) {
          const int r = e % CW_, c = e / CW_;
          if (r >= w && r >= c) P[r + c * LD] = r == c ? 1.0 : 0.0;
        }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // (the first time: the right-hand sides too)
      for (int e = tid; e < nrhs * CW_; e += NT) {
        const int q = e / CW_, c = e % CW_;
        P[RB + q + c * LD] = c < w ? sR[j + c + q * LDR] : 0.0;
      }
      __syncthreads();
      // ---- panel, eight columns a step: warp 0 factors the 8 x 8 block and
      // solves the rest of the diagonal block's rows; the rows below follow
      // after the barrier, beside its next step
      const int row = CW_ + (warp - 1) * 32 + lane;
      for (int s = 0; s < CW_; s += 8) {
        double x[8];
        if (warp == 0) {
          row_minus<LD>(P, lane, s, x);
          if (lane >= s) store8<LD>(P, lane, s, x);
          __syncwarp();
          double l[36], ri[8];
          const int f = chol8_load_factor(P + s + s * LD, LD, l, ri);
          chol8_solve(l, ri, x);
          __syncwarp();
          if (lane >= s) store8<LD>(P, lane, s, x);
          if (lane == 0) {
            if (f >= 0 && s + f < w && s_fail < 0) s_fail = s + f;
#pragma unroll
            for (int k = 0; k < 8; ++k) rinv[s + k] = ri[k];
          }
        } else if (row < RB + nrhs) {
          row_minus<LD>(P, row, s, x);
        }
        __syncthreads();
        if (warp != 0 && row < RB + nrhs) {
          row_solve<LD>(P, s, rinv, x);
          store8<LD>(P, row, s, x);
          // at most eight rows, in the first panel of the largest orders
          if (const int r2 = row + (NW - 1) * 32; r2 < RB + nrhs) {
            row_minus<LD>(P, r2, s, x);
            row_solve<LD>(P, s, rinv, x);
            store8<LD>(P, r2, s, x);
          }
        }
      }
      __syncthreads();
      if (s_fail >= 0) {
        // as far as the leading minor goes: the diagonal block's columns before
        // the failing one, and what is left of its others
        const int f = s_fail;
        for (int e = tid; e < w * w; e += NT) {
          const int r = e % w, c = e / w;
          if (r < c) continue;
          double* d = G + (long)(j + r) + (long)(j + c) * ld;
          if (c < f) {
            *d = P[r + c * LD];
          } else {
            double v = *d;
            for (int k = 0; k < f; ++k) v = fma(-P[r + k * LD], P[c + k * LD], v);
            *d = v;
          }
        }
        fail = j + f;
        break;
      }
      // ---- back to memory, and the right-hand sides' entries
      for (int c = warp; c < w; c += NW)
        for (int r = c + lane; r < R; r += 32) G[(long)(j + r) + (long)(j + c) * ld] = P[r + c * LD];
      for (int e = tid; e < nrhs * w; e += NT) {
        const int q = e / w, c = e % w;
        sR[j + c + q * LDR] = P[RB + q + c * LD];
      }
      if (R <= CW_) continue;  // the last panel
      // ---- A22 -= L21 L21^T: tiles of 16 rows x 32 columns on or below the
      // diagonal, then one strip of the right-hand sides' rows
      const int R2 = R - CW_;
      const int tr = (R2 + 15) / 16, tc = (R2 + 31) / 32;
      int c32 = 0, e = warp;  // tile e of column tile c32 (row tiles 2 c32 ..)
      for (;; e += NW) {
        while (c32 < tc && e >= tr - 2 * c32) e -= tr - 2 * c32++;
        if (c32 == tc) break;
        const int r0 = (2 * c32 + e) * 16, c0 = c32 * 32;
        double* C = G + (long)(j + CW_) + (long)(j + CW_) * ld;
        double v[2][4][2], d[2][4][2];  // the tile's entries arrive during the products
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int rw = r0 + 8 * i + g, col = c0 + 8 * c + 2 * t + h;
              v[i][c][h] = (rw < R2 && col <= rw) ? C[rw + (long)col * ld] : 0.0;
              d[i][c][h] = 0.0;
            }
        // rows past the matrix: whatever P holds there, never stored
        const double* pa = P + CW_ + r0 + g + t * LD;
        const double* pb = P + CW_ + c0 + g + t * LD;
#pragma unroll
        for (int k = 0; k < CW_; k += 4) {
          const double a0 = pa[k * LD], a1 = pa[8 + k * LD];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const double b = pb[8 * c + k * LD];
            dmma_884(d[0][c][0], d[0][c][1], a0, b);
            dmma_884(d[1][c][0], d[1][c][1], a1, b);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int rw = r0 + 8 * i + g, col = c0 + 8 * c + 2 * t + h;
              if (rw < R2 && col <= rw) C[rw + (long)col * ld] = v[i][c][h] - d[i][c][h];
            }
      }
      // the right-hand sides' rows: one row tile
      for (int c0 = e * 32; nrhs > 0 && c0 < R2; c0 += NW * 32) {
        double d[4][2];
#pragma unroll
        for (int c = 0; c < 4; ++c) d[c][0] = d[c][1] = 0.0;
        const double* pa = P + CW_ + R2 + g + t * LD;
        const double* pb = P + CW_ + c0 + g + t * LD;
#pragma unroll
        for (int k = 0; k < CW_; k += 4)
#pragma unroll
          for (int c = 0; c < 4; ++c) dmma_884(d[c][0], d[c][1], pa[k * LD], pb[8 * c + k * LD]);
        if (g < nrhs)
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int col = c0 + 8 * c + 2 * t + h;
              if (col < R2) sR[j + CW_ + col + g * LDR] -= d[c][h];
            }
      }
      __syncthreads();  // the next panel reads the update; P is reused
    }
    __syncthreads();
    if (tid == 0) a.info[mi] = fail;
    // log-determinant (fixed order: lane-strided partial sums, shuffle tree)
    if (a.logdet && warp == 0) {
      double sl = 0.0;
      if (fail < 0)
        for (int i = lane; i < n; i += 32) sl += log(G[(long)i + (long)i * ld]);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) sl += __shfl_xor_sync(0xffffffffu, sl, off);
      if (lane == 0) a.logdet[mi] = fail < 0 ? sl : __longlong_as_double(0x7ff8000000000000ll);
    }
    // ---- backward substitution L^T x = y
    if (nrhs > 0 && fail < 0) {
      double* sD = P;                       // [2] diagonal blocks, L(r, c) at r + 33 c
      double* sS = P + 2 * CW_ * (CW_ + 1);  // [NW / 4][CRHS][32] partial products
      const int last = (n - 1) / CW_ * CW_;
      __syncthreads();
      for (int e = tid; e < CW_ * CW_; e += NT) {
        const int r = e % CW_, c = e / CW_, w = n - last;
        sD[r + c * 33] = r < w && c <= r ? G[(long)(last + r) + (long)(last + c) * ld] : (r == c ? 1.0 : 0.0);
      }
      for (int b0 = last, i = 0; b0 >= 0; b0 -= CW_, i ^= 1) {
        if (b0 > 0)  // the next diagonal block
          for (int e = tid; e < CW_ * CW_; e += NT) {
            const int r = e % CW_, c = e / CW_;
            if (c <= r)
              cp_async8(sD + (i ^ 1) * CW_ * (CW_ + 1) + r + c * 33,
                        G + (long)(b0 - CW_ + r) + (long)(b0 - CW_ + c) * ld);
          }
        // L(below, block)^T times the solved rows: warp & 3 takes eight of the
        // columns, warp >> 2 a share of the rows
        const int cg = 8 * (warp & 3), ks = warp >> 2;
        if (b0 < last) {
          double d0 = 0.0, d1 = 0.0;
          const double* gb = G + (long)(b0 + cg + g) * ld + t;
          const double* ra = sR + t + g * LDR;
          for (int k = b0 + CW_ + 4 * ks; k < n; k += 8 * NW) {
            double av[8], bv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int kk = k + u * NW;
              const bool in = kk + t < n;
              bv[u] = in ? gb[kk] : 0.0;
              av[u] = in ? ra[kk] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) dmma_884(d0, d1, av[u], bv[u]);
          }
          double* o = sS + (ks * CRHS + g) * CW_ + cg + 2 * t;
          o[0] = d0;
          o[1] = d1;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const int w = min(CW_, n - b0);
        const double* D = sD + i * CW_ * (CW_ + 1);
        for (int q = warp; q < nrhs; q += NW) {
          double y = lane < w ? sR[b0 + lane + q * LDR] : 0.0;
          if (b0 < last) {
            double u = 0.0;
#pragma unroll
            for (int k = 0; k < NW / 4; ++k) u += sS[(k * CRHS + q) * CW_ + lane];
            y -= u;
          }
          const double rv = 1.0 / D[lane + lane * 33];
          double sol = 0.0;
#pragma unroll
          for (int s = CW_ - 8; s >= 0; s -= 8) {  // eight entries in every lane, then the lane's own
            double x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = __shfl_sync(0xffffffffu, y, s + k);
#pragma unroll
            for (int k = 7; k >= 0; --k) {
              x[k] *= __shfl_sync(0xffffffffu, rv, s + k);
#pragma unroll
              for (int c = 0; c < k; ++c) x[c] = fma(-D[s + k + (s + c) * 33], x[k], x[c]);
              if (lane == s + k) sol = x[k];
            }
#pragma unroll
            for (int k = 7; k >= 0; --k) y = fma(-D[s + k + lane * 33], x[k], y);  // only lanes below s count
          }
          if (lane < w) {
            sR[b0 + lane + q * LDR] = sol;
            a.B[mi][(long)(b0 + lane) + (long)q * a.ldb[mi]] = sol;
          }
        }
        __syncthreads();
      }
    }
  }
}

template <int NT>
int chb_launch(const BatchArgs<double>& a, int grid, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    FB_CK(cudaFuncSetAttribute(chol_batched_f64_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)ChB<NT>::SMEM));
    attr = true;
  }
  const int ps = prof_begin(st);
  chol_batched_f64_kernel<NT><<<grid, NT, ChB<NT>::SMEM, st>>>(a);
  prof_end(ps, st, PROF_OTHER, 0.0);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

}  // namespace

// Orders up to 512; a.order: `mid` matrices above order 256 first; a.counter:
// two words.
int batched_chol_f64(const BatchArgs<double>& a, int mid, cudaStream_t st) {
  const int sms = ctx().num_sms;
  BatchArgs<double> b = a;
  b.count = mid;
  if (mid > 0 && chb_launch<512>(b, std::min(sms, mid), st) != FLA_SUCCESS) return FLA_FAILURE;
  b.count = a.count - mid;
  b.order = a.order + mid;
  b.counter = a.counter + 1;
  if (b.count > 0 && chb_launch<256>(b, std::min(2 * sms, b.count), st) != FLA_SUCCESS) return FLA_FAILURE;
  return FLA_SUCCESS;
}

}  // namespace fb
