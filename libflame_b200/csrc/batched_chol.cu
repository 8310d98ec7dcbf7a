// Batched FP64 Cholesky (+ solves, log-determinants) for many small matrices
// of uneven sizes, orders up to 512: one CTA per matrix, matrices from an
// atomic counter in a host-chosen order (largest first).
//
// Semantics of FLA_Chol per matrix (src/lapack/dec/chol/front/flamec/
// FLA_Chol.c:16-29): lower triangle only, stopping at the first pivot that is
// not > 0 (NaN included), its zero-based column reported; a matrix that fails
// keeps its right-hand sides.
//
// Right-looking in panels of 32 columns, in place (the matrices of the
// resident CTAs stay in L2):
//   panel   the block column in shared memory; one warp factors its 32 x 32
//           diagonal block and publishes each column, the other warps solve
//           the rows below one column behind it (chol_leaf.cuh);
//   update  A22 -= L21 L21^T (lower) on the FP64 tensor cores, 16 x 32 warp
//           tiles, both operands from the panel in shared memory.
// The right-hand sides are rows below the matrix (kept in shared memory), so
// the forward substitution comes with the factorization.  Bound by the pivot
// chain of the panels (about 0.13 us a column) and, for the large orders, the
// FP64 rate.  Orders up to 256 run in CTAs of 256 threads, two per SM, so that
// one matrix's chain overlaps the other's updates; 257 to 512 in CTAs of 512.
// Measured: 2500 matrices, n uniform in 8..512, 4 right-hand sides: 11.9 ms
// left-looking with one CTA of 512 threads per SM (chol_batched_dmma_kernel,
// which keeps the orders above 512), 4.5 ms in this form.
#include <algorithm>

#include "batched.h"
#include "chol_leaf.cuh"
#include "common.h"

namespace fb {

namespace {

constexpr int CW_ = CHOL_IB;      // panel width
constexpr int CRHS = 8;           // right-hand sides

template <int NT>
struct ChB {
  static constexpr int NW = NT / 32;
  static constexpr int LD = NT + 20;        // rows of the panel: NT, the right-hand sides, a tile's rest; = 4 mod 16
  static constexpr int LDR = NT;            // right-hand side q at sR[q * LDR]
  static constexpr size_t SMEM = sizeof(double) * ((size_t)LD * CW_ + (size_t)CRHS * LDR + 2 * CW_ + CRHS * CW_);
  static constexpr int MINB = NT == 256 ? 2 : 1;
};

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

template <int NT>
__global__ void __launch_bounds__(NT, ChB<NT>::MINB) chol_batched_f64_kernel(BatchArgs<double> a) {
  using B = ChB<NT>;
  constexpr int NW = B::NW, LD = B::LD, LDR = B::LDR;
  extern __shared__ __align__(16) double chb_sm[];
  double* P = chb_sm;                      // panel: row r (from the panel's first), column c at P[r + c * LD]
  double* sR = P + (size_t)LD * CW_;       // right-hand sides
  double* s_rinv = sR + CRHS * LDR;        // [2][32], by panel parity
  double* sx = s_rinv + 2 * CW_;           // [CRHS][32]
  __shared__ int s_next, s_fail, s_cnt;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_next = atomicAdd(a.counter, 1);
      s_fail = -1;
      s_cnt = 0;
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
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // (the first time: the right-hand sides too)
      for (int e = tid; e < nrhs * CW_; e += NT) {
        const int q = e / CW_, c = e % CW_;
        P[RB + q + c * LD] = c < w ? sR[j + c + q * LDR] : 0.0;
      }
      __syncthreads();
      // ---- panel; the counter runs on over the panels
      double* rinv = s_rinv + ((j / CW_) & 1) * CW_;
      if (warp == 0) {
        potrf_diag32<LD>(P, 0, w, lane, rinv, &s_cnt, j, &s_fail);
      } else {
        for (int r = CW_ + (warp - 1) * 32 + lane; r < RB + nrhs; r += (NW - 1) * 32)
          potrf_row<LD>(P, 0, r, rinv, &s_cnt, j, a.err);
      }
      __syncthreads();
      if (s_fail >= 0) {
        fail = j + s_fail;
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
      const int strips = nrhs > 0 ? tc : 0;
      for (int e = warp; e < tr * tc + strips; e += NW) {
        const bool rhs = e >= tr * tc;
        const int r0 = rhs ? R2 : (e % tr) * 16, c0 = (rhs ? e - tr * tc : e / tr) * 32;
        if (!rhs && r0 + 15 < c0) continue;
        double d[2][4][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) d[i][c][0] = d[i][c][1] = 0.0;
        const double* pa = P + CW_ + r0 + g + t * LD;
        const double* pb = P + CW_ + c0 + g + t * LD;
        const bool two = !rhs;  // eight right-hand sides: one row tile
#pragma unroll 4
        for (int k = 0; k < CW_; k += 4) {
          const double a0 = pa[k * LD], a1 = two ? pa[8 + k * LD] : 0.0;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            // column tiles past the matrix: any finite or garbage row of P, never stored
            const double b = c0 + 8 * c < R2 ? pb[8 * c + k * LD] : 0.0;
            dmma_884(d[0][c][0], d[0][c][1], a0, b);
            if (two) dmma_884(d[1][c][0], d[1][c][1], a1, b);
          }
        }
        if (rhs) {
          if (g < nrhs)
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int col = c0 + 8 * c + 2 * t + h;
                if (col < R2) sR[j + CW_ + col + g * LDR] -= d[0][c][h];
              }
        } else {
          double* C = G + (long)(j + CW_) + (long)(j + CW_) * ld;
          double v[2][4][2];
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int row = r0 + 8 * i + g, col = c0 + 8 * c + 2 * t + h;
                v[i][c][h] = (row < R2 && col <= row) ? C[row + (long)col * ld] : 0.0;
              }
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int row = r0 + 8 * i + g, col = c0 + 8 * c + 2 * t + h;
                if (row < R2 && col <= row) C[row + (long)col * ld] = v[i][c][h] - d[i][c][h];
              }
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
      double* sD = P;  // diagonal block, sD[r + c * 33]
      for (int b0 = (n - 1) / CW_ * CW_; b0 >= 0; b0 -= CW_) {
        const int w = min(CW_, n - b0);
        __syncthreads();
        for (int e = tid; e < CW_ * CW_; e += NT) {
          const int r = e % CW_, c = e / CW_;
          sD[r + c * 33] = r < w && c <= r ? G[(long)(b0 + r) + (long)(b0 + c) * ld] : (r == c ? 1.0 : 0.0);
        }
        __syncthreads();
        for (int q = warp; q < nrhs; q += NW) {
          double y = lane < w ? sR[b0 + lane + q * LDR] : 0.0;
          const double rv = 1.0 / sD[lane + lane * 33];
          for (int s = w - 1; s >= 0; --s) {
            const double x = __shfl_sync(0xffffffffu, y * rv, s);
            if (lane == s) y = x;
            else if (lane < s) y = fma(-sD[s + lane * 33], x, y);
          }
          sx[q * CW_ + lane] = y;
          if (lane < w) a.B[mi][(long)(b0 + lane) + (long)q * a.ldb[mi]] = y;
        }
        __syncthreads();
        for (int r = tid; r < b0; r += NT) {
          const double* p = G + (long)b0 + (long)r * ld;
          double u[CW_];
#pragma unroll
          for (int s = 0; s < CW_; ++s) u[s] = s < w ? p[s] : 0.0;
          for (int q = 0; q < nrhs; ++q) {
            double y0 = sR[r + q * LDR], y1 = 0.0;
#pragma unroll
            for (int s = 0; s < CW_; s += 2) {
              y0 = fma(-u[s], sx[q * CW_ + s], y0);
              y1 = fma(-u[s + 1], sx[q * CW_ + s + 1], y1);
            }
            sR[r + q * LDR] = y0 + y1;
          }
        }
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
