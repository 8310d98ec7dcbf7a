// X := X inv(L)^T for a tall block X (m x b, column-major) and a lower
// triangular L of order b <= 128: the triangular solves of the panels.
//
//   Cholesky: A21 := A21 inv(L11)^T (FLA_Chol_l_blk_var3.c), non-unit L11,
//             column-major, FP64 or (low-precision factors) FP32 X;
//   LU on A^T: U12 := inv(L11) A12 (FLA_LU_piv_blk_var5.c), unit L11; on the
//             transposed storage U12^T is X and row i of L11 a contiguous
//             column of A^T.
//
// By steps of 16 columns, the reference's order within a step: a thread per row
// solves them by forward substitution in registers (dtrsm's R,L,T,N case), the
// products with the columns beyond are subtracted on the FP64 tensor cores:
// first those the next step needs, the rest beside its substitution.  A CTA
// holds the triangle and ROWS rows of X; fewer rows per CTA when there are few
// rows, so that they spread over the SMs.  Bound by the latency of the load and
// the chain of steps; sixteen columns, because a step's 120 FMAs then just fill
// the latency of its own chain of sixteen.
// Substitution rather than products with inverted diagonal blocks: the error of
// those grows with the condition of the block (n = 512, squared-exponential
// kernel, nugget 1e-9: ||A - L L^T|| / ||A|| 2.6e-15 with 32 x 32 inverses,
// 1.5e-16 so; an LU whose 32 x 32 blocks are near -1 below the diagonal 1.1e-8
// and 1.2e-16), and an infinite entry spoils columns before its own.  FLA_Chol
// n = 1024 takes 327 us with inverses, 335 us so (eight solves); FLA_LU_piv
// n = 3001 6.24 ms both ways.  (A shuffle per column, a warp per row group:
// 896 x 128 16.2 us against 10.2 with the inverses; a row per thread by 32
// columns 17.8.)
#include <algorithm>

#include "common.h"
#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int RB = 128;           // widest triangle
constexpr int RIB = 16;           // columns per substitution step
constexpr int RLD = RB + 4;       // = 4 mod 16: conflict-free DMMA fragments
constexpr int R_THREADS = 256;

template <int ROWS>
constexpr int rlt_ldx() { return ROWS + 4; }  // = 4 mod 16
template <int ROWS>
size_t rlt_smem(int b) {
  const int bp = (b + RIB - 1) / RIB * RIB;
  return sizeof(double) * ((size_t)bp * RLD + (size_t)bp * rlt_ldx<ROWS>() + RB);
}

// X(:, c) -= X(:, kb..kb+15) L(c, kb..kb+15)^T for the 8-column tiles from c_lo
// up to c_hi, the tiles of 8 rows dealt to nw warps, w the calling one.
template <int ROWS>
__device__ __forceinline__ void rlt_update(const double* sL, double* sX, int kb, int c_lo, int c_hi, int w, int nw, int lane) {
  constexpr int LDX = rlt_ldx<ROWS>(), TI = ROWS / 8;
  const int g = lane >> 2, t = lane & 3;
  for (int e = w; e < TI * ((c_hi - c_lo) >> 3); e += nw) {
    const int r = 8 * (e % TI), c = c_lo + 8 * (e / TI);
    const double* pa = sX + r + g + (kb + t) * LDX;
    const double* pb = sL + c + g + (kb + t) * RLD;
    double* o = sX + r + g + (c + 2 * t) * LDX;
    const double o0 = o[0], o1 = o[LDX];
    double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};  // halves of the sixteen, in order
#pragma unroll
    for (int k = 0; k < RIB / 2; k += 4) {
      dmma_884(d0[0], d0[1], pa[k * LDX], pb[k * RLD]);
      dmma_884(d1[0], d1[1], pa[(k + RIB / 2) * LDX], pb[(k + RIB / 2) * RLD]);
    }
    o[0] = o0 - (d0[0] + d1[0]);
    o[LDX] = o1 - (d0[1] + d1[1]);
  }
}

// x := x inv(D)^T for a row x of RIB entries, D the diagonal block at D (ld
// RLD), its reciprocal pivots in rinv.
template <bool UNIT>
__device__ __forceinline__ void rlt_solve(const double* D, const double* rinv, double (&x)[RIB]) {
#pragma unroll
  for (int k = 0; k < RIB; ++k) {
    if (!UNIT) x[k] *= rinv[k];
    if (k % 2 == 0) x[k + 1] = fma(-D[k + 1 + k * RLD], x[k], x[k + 1]);
#pragma unroll
    for (int c = (k + 2) & ~1; c < RIB; c += 2) {
      const double2 v = *reinterpret_cast<const double2*>(D + c + k * RLD);
      x[c] = fma(-v.x, x[k], x[c]);
      x[c + 1] = fma(-v.y, x[k], x[c + 1]);
    }
  }
}

// UNIT: unit L with L(i, j) at Ls[j + i ld]; else non-unit, L(i, j) at
// Ls[i + j ld].  X(r, c) at X[r + c ldx].  Returns at once when *guard holds
// a failing column below guard_limit.
template <int ROWS, bool UNIT, typename TX>
__global__ void __launch_bounds__(R_THREADS, 1) rlt_kernel(const double* __restrict__ Ls, long ld, TX* __restrict__ X,
                                                        long ldx, int b, long m, const int* guard, int guard_limit) {
  chain_begin();
  constexpr int LDX = rlt_ldx<ROWS>();
  extern __shared__ __align__(16) double rlt_sm[];
  if (guard && *((volatile const int*)guard) < guard_limit) return;
  const int bp = (b + RIB - 1) / RIB * RIB;
  double* sL = rlt_sm;               // L(i, j) at sL[i + j * RLD]
  double* sX = sL + bp * RLD;       // X(r, c) at sX[r + c * LDX]
  double* sR = sX + bp * LDX;       // reciprocal pivots
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long r0 = (long)blockIdx.x * ROWS;
  const int rows = (int)(m - r0 < ROWS ? m - r0 : ROWS);
  // the triangle, along its contiguous index; past b the identity
  for (int o = warp; o < b; o += R_THREADS / 32) {
    if (UNIT) {  // row o: entries e < o
      for (int e = lane; e < o; e += 32) cp_async8(sL + o + e * RLD, Ls + e + (long)o * ld);
    } else {     // column o: entries e >= o
      for (int e = o + lane; e < b; e += 32) cp_async8(sL + e + o * RLD, Ls + e + (long)o * ld);
    }
  }
  if constexpr (sizeof(TX) == 8) {
    for (int e = tid; e < ROWS * b; e += R_THREADS) {
      const int r = e % ROWS, c = e / ROWS;
      if (r < rows) cp_async8(sX + r + c * LDX, (const double*)X + r0 + r + (long)c * ldx);
    }
  } else {
#pragma unroll 8
    for (int e = tid; e < ROWS * b; e += R_THREADS) {
      const int r = e % ROWS, c = e / ROWS;
      sX[r + c * LDX] = r < rows ? (double)X[r0 + r + (long)c * ldx] : 0.0;
    }
  }
  if (b < bp) {  // rows of the triangle and columns of X past b
    for (int e = tid; e < bp * (bp - b); e += R_THREADS) sL[b + e % (bp - b) + e / (bp - b) * RLD] = 0.0;
    for (int e = tid; e < ROWS * (bp - b); e += R_THREADS) sX[e % ROWS + (b + e / ROWS) * LDX] = 0.0;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (!UNIT) {
    for (int j = tid; j < bp; j += R_THREADS) sR[j] = j < b ? 1.0 / sL[j + j * RLD] : 1.0;
    __syncthreads();
  }
  // row warps: a thread per row; the others subtract the products, with few
  // rows without the one on the row warp's sub-partition
  constexpr int RW = (ROWS + 31) / 32;
  constexpr int UW = ROWS <= 32 ? 6 : R_THREADS / 32 - RW;
  const int uw = ROWS <= 32 ? (warp & 3) - 1 + 3 * (warp >> 2) : warp - RW;  // UW update warps
  const bool upd = ROWS <= 32 ? (warp & 3) != 0 : warp >= RW;
  for (int kb = 0; kb < b; kb += RIB) {
    if (warp < RW) {
      if (tid < ROWS) {
        double x[RIB];
        double* row = sX + tid + kb * LDX;
#pragma unroll
        for (int c = 0; c < RIB; ++c) x[c] = row[c * LDX];
        rlt_solve<UNIT>(sL + kb * (1 + RLD), sR + kb, x);
#pragma unroll
        for (int c = 0; c < RIB; ++c) row[c * LDX] = x[c];
      }
    } else if (upd && kb > 0) {
      rlt_update<ROWS>(sL, sX, kb - RIB, kb + RIB, bp, uw, UW, lane);
    }
    __syncthreads();
    if (kb + RIB >= b) break;
    rlt_update<ROWS>(sL, sX, kb, kb + RIB, kb + 2 * RIB, warp, R_THREADS / 32, lane);
    __syncthreads();
  }
  chain_next();
#pragma unroll 4
  for (int e = tid; e < ROWS * b; e += R_THREADS) {
    const int r = e % ROWS, c = e / ROWS;
    if (r < rows) X[r0 + r + (long)c * ldx] = (TX)sX[r + c * LDX];
  }
}

template <int ROWS, bool UNIT, typename TX>
void rlt_launch(const double* L, long ld, TX* X, long ldx, int b, long m, const int* guard, int guard_limit,
                cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(rlt_kernel<ROWS, UNIT, TX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rlt_smem<ROWS>(RB));
    attr = true;
  }
  FB_LAUNCH(launch_chain(rlt_kernel<ROWS, UNIT, TX>, dim3((unsigned)((m + ROWS - 1) / ROWS)), dim3(R_THREADS), rlt_smem<ROWS>(b), st,
        L, ld, X, ldx, b, m, guard, guard_limit));
}

// Rows per CTA: the fewest that leave one wave (shared memory allows one CTA per
// SM with a 128-column triangle, two with a 64-column one).
template <bool UNIT, typename TX>
int rlt_any(const double* L, long ld, TX* X, long ldx, int b, long m, const int* guard, int guard_limit,
            cudaStream_t st) {
  if (m <= 0 || b <= 0) return FLA_SUCCESS;
  if (b > RB) {
    set_last_error("triangular solve: triangle wider than 128");
    return FLA_FAILURE;
  }
  const long wave = (long)ctx().num_sms * (b <= 64 ? 2 : 1);
  const int ps = prof_begin(st);
  if (m <= 16 * wave) rlt_launch<16, UNIT, TX>(L, ld, X, ldx, b, m, guard, guard_limit, st);
  else if (m <= 32 * wave) rlt_launch<32, UNIT, TX>(L, ld, X, ldx, b, m, guard, guard_limit, st);
  else rlt_launch<64, UNIT, TX>(L, ld, X, ldx, b, m, guard, guard_limit, st);
  prof_end(ps, st, PROF_TRSM, (double)m * b * b);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

}  // namespace

int trsm_rlt_subst(const double* L, double* X, long ld, int b, long m, const int* guard, int guard_limit,
                   cudaStream_t st) {
  return rlt_any<false, double>(L, ld, X, ld, b, m, guard, guard_limit, st);
}

int trsm_rlt_subst_f32(const double* L, long ldl, float* X, long ldx, int b, long m, const int* guard,
                       int guard_limit, cudaStream_t st) {
  return rlt_any<false, float>(L, ldl, X, ldx, b, m, guard, guard_limit, st);
}

// U12 := inv(L11) A12 for ncols columns, any b: blocks of 128 rows, the rows
// below each updated by a GEMM.
int u12_subst(const double* Ls, double* X, long ld, int b, long ncols, cudaStream_t st) {
  if (ncols <= 0 || b <= 0) return FLA_SUCCESS;
  for (int r0 = 0; r0 < b; r0 += RB) {
    const int bb = std::min(RB, b - r0);
    double* Y = X + (long)r0 * ld;
    if (rlt_any<true, double>(Ls + r0 + (long)r0 * ld, ld, Y, ld, bb, ncols, nullptr, 0, st) != FLA_SUCCESS)
      return FLA_FAILURE;
    const int rest = b - r0 - bb;
    // U12^T[:, r0+bb:] -= U12^T[:, r0:r0+bb] L11^T[r0:r0+bb, r0+bb:]
    if (rest > 0 && gemm_f64(st, false, false, ncols, rest, bb, -1.0, Y, ld, Ls + r0 + (long)(r0 + bb) * ld, ld,
                             1.0, X + (long)(r0 + bb) * ld, ld) != FLA_SUCCESS)
      return FLA_FAILURE;
  }
  return FLA_SUCCESS;
}

}  // namespace fb
