// X := X inv(L)^T for a tall block X (m x b, column-major) and a lower
// triangular L of order b <= 128: the triangular solves of the panels.
//
//   Cholesky: A21 := A21 inv(L11)^T (FLA_Chol_l_blk_var3.c), non-unit L11,
//             column-major, FP64 or (low-precision factors) FP32 X;
//   LU on A^T: U12 := inv(L11) A12 (FLA_LU_piv_blk_var5.c), unit L11; on the
//             transposed storage U12^T is X and row i of L11 a contiguous
//             column of A^T.
//
// By 32-column blocks: X_k := A_k inv(L_kk)^T, then the products of block k
// are subtracted from the columns to its right, all on the FP64 tensor cores.
// The inverses of the 32 x 32 diagonal blocks (zero above the diagonal) take
// their place in shared memory first: eight warps invert the 16 x 16 blocks
// by forward substitution, one column per lane, and each 32 x 32 one is
// completed by I21 = -I22 (L21 I11).  A CTA holds the triangle and ROWS rows
// of X; fewer rows per CTA when there are few rows, so that they spread over
// the SMs.  Bound by the latency of the load, the 16 dependent steps of the
// small inverses and four pairs of products.
// Measured against forward substitution with a shuffle per column (a warp
// per row group): 896 x 128 16.2 -> 10.2 us, the LU's joins (up to 128 x 128) 9.8 -> 7.2 us on
// average; 8000 x 128 takes 18 us, less than inv(L11), a copy and a product.
// (Substitution with a row per thread by 32-column blocks took 17.8 us: one
// warp's 496 dependent loads and FMAs per block.)
#include <algorithm>

#include "common.h"
#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int RB = 128;           // widest triangle
constexpr int RIB = 32;           // columns per substitution step
constexpr int RLD = RB + 4;       // = 4 mod 16: conflict-free DMMA fragments
constexpr int R_THREADS = 256;

template <int ROWS>
constexpr int rlt_ldx() { return ROWS + 4; }  // = 4 mod 16
template <int ROWS>
size_t rlt_smem(int b) {
  const int b32 = (b + RIB - 1) / RIB * RIB;
  return sizeof(double) * ((size_t)b32 * RLD + (size_t)b32 * rlt_ldx<ROWS>() + RB);
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// X(:, c_lo + 8 j) -= X(:, kb..kb+31) L(c, kb..kb+31)^T for ntj 8-column
// tiles, the ROWS/8 x ntj tiles dealt to the warps.
template <int ROWS>
__device__ __forceinline__ void rlt_update(const double* sL, double* sX, int kb, int c_lo, int ntj, int w, int lane) {
  constexpr int LDX = rlt_ldx<ROWS>(), TI = ROWS / 8;
  const int g = lane >> 2, t = lane & 3;
  for (int e = w; e < TI * ntj; e += R_THREADS / 32) {
    const int r = 8 * (e % TI), c = c_lo + 8 * (e / TI);
    const double* pa = sX + r + g + (kb + t) * LDX;
    const double* pb = sL + c + g + (kb + t) * RLD;
    double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < RIB; k += 8) {
      dmma_884(d0[0], d0[1], pa[k * LDX], pb[k * RLD]);
      dmma_884(d1[0], d1[1], pa[(k + 4) * LDX], pb[(k + 4) * RLD]);
    }
    double* o = sX + r + g + (c + 2 * t) * LDX;
    o[0] -= d0[0] + d1[0];
    o[LDX] -= d0[1] + d1[1];
  }
}

// The 16 x 16 diagonal block at D := its inverse, zero above the diagonal.
template <bool UNIT>
__device__ __forceinline__ void rlt_invert16(double* D, const double* rinv, int lane) {
  const int c = lane & 15;
  double x[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) x[r] = r == c ? 1.0 : 0.0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (!UNIT) x[j] *= rinv[j];
    double l[16];
#pragma unroll
    for (int r = (j + 1) & ~1; r < 16; r += 2) {
      const double2 v = *reinterpret_cast<const double2*>(D + r + j * RLD);
      l[r] = v.x;
      l[r + 1] = v.y;
    }
#pragma unroll
    for (int r = j + 1; r < 16; ++r) x[r] = fma(-l[r], x[j], x[r]);
  }
  __syncwarp();
  if (lane < 16)
#pragma unroll
    for (int r = 0; r < 16; ++r) D[r + c * RLD] = r >= c ? x[r] : 0.0;
}

// Z := sgn Y W for 16 x 16 blocks in shared memory (ld RLD), by one warp; Z
// may not overlap Y or W.
__device__ __forceinline__ void rlt_mul16(const double* Y, const double* Wm, double* Z, double sgn, int lane) {
  const int g = lane >> 2, t = lane & 3;
  double d[2][2][2] = {};
#pragma unroll
  for (int k = 0; k < 16; k += 4)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
        dmma_884(d[i][j][0], d[i][j][1], Y[8 * i + g + (k + t) * RLD], Wm[k + t + (8 * j + g) * RLD]);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) Z[8 * i + g + (8 * j + 2 * t + e) * RLD] = sgn * d[i][j][e];
}

// UNIT: unit L with L(i, j) at Ls[j + i ld]; else non-unit, L(i, j) at
// Ls[i + j ld].  X(r, c) at X[r + c ldx].  Returns at once when *guard holds
// a failing column below guard_limit.
template <int ROWS, bool UNIT, typename TX>
__global__ void __launch_bounds__(R_THREADS) rlt_kernel(const double* __restrict__ Ls, long ld, TX* __restrict__ X,
                                                        long ldx, int b, long m, const int* guard, int guard_limit) {
  chain_begin();
  constexpr int LDX = rlt_ldx<ROWS>();
  extern __shared__ __align__(16) double rlt_sm[];
  if (guard && *((volatile const int*)guard) < guard_limit) return;
  const int b32 = (b + RIB - 1) / RIB * RIB, b8 = (b + 7) & ~7;
  double* sL = rlt_sm;               // L(i, j) at sL[i + j * RLD]
  double* sX = sL + b32 * RLD;       // X(r, c) at sX[r + c * LDX]
  double* sR = sX + b32 * LDX;       // reciprocal pivots
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
  if (b < b32) {  // rows of the triangle and columns of X past b
    for (int e = tid; e < b32 * (b32 - b); e += R_THREADS) sL[b + e % (b32 - b) + e / (b32 - b) * RLD] = 0.0;
    for (int e = tid; e < ROWS * (b32 - b); e += R_THREADS) sX[e % ROWS + (b + e / ROWS) * LDX] = 0.0;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (!UNIT) {
    for (int j = tid; j < b32; j += R_THREADS) sR[j] = j < b ? 1.0 / sL[j + j * RLD] : 1.0;
    __syncthreads();
  }
  // inverses of the diagonal blocks, in place
  if (16 * warp < b32) rlt_invert16<UNIT>(sL + 16 * warp * (1 + RLD), sR + 16 * warp, lane);
  __syncthreads();
  if (RIB * warp < b32) {
    double* D = sL + RIB * warp * (1 + RLD);
    double* Tm = D + 16 * RLD;  // the block's upper right quarter, for L21 I11
    rlt_mul16(D + 16, D, Tm, 1.0, lane);
    __syncwarp();
    rlt_mul16(D + 16 * (1 + RLD), Tm, D + 16, -1.0, lane);
    __syncwarp();
    for (int e = lane; e < 256; e += 32) Tm[(e & 15) + (e >> 4) * RLD] = 0.0;
  }
  __syncthreads();
  constexpr int TPW = (ROWS / 8) * (RIB / 8) / (R_THREADS / 32);  // tiles of X_k per warp
  const int g = lane >> 2, t = lane & 3;
  for (int kb = 0; kb < b; kb += RIB) {
    // X_k := A_k inv(L_kk)^T: tile (ri, cj), k up to the end of column tile cj
    double x[TPW][2];
#pragma unroll
    for (int u = 0; u < TPW; ++u) {
      const int e = warp + u * (R_THREADS / 32);
      const int r = 8 * (e % (ROWS / 8)), c = 8 * (e / (ROWS / 8));
      const double* pa = sX + r + g + (kb + t) * LDX;
      const double* pb = sL + kb + c + g + (kb + t) * RLD;
      double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
      for (int k = 0; k <= c; k += 8) {
        dmma_884(d0[0], d0[1], pa[k * LDX], pb[k * RLD]);
        dmma_884(d1[0], d1[1], pa[(k + 4) * LDX], pb[(k + 4) * RLD]);
      }
      x[u][0] = d0[0] + d1[0];
      x[u][1] = d0[1] + d1[1];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < TPW; ++u) {
      const int e = warp + u * (R_THREADS / 32);
      const int r = 8 * (e % (ROWS / 8)), c = 8 * (e / (ROWS / 8));
      double* o = sX + r + g + (kb + c + 2 * t) * LDX;
      o[0] = x[u][0];
      o[LDX] = x[u][1];
    }
    __syncthreads();
    if (kb + RIB >= b8) break;
    rlt_update<ROWS>(sL, sX, kb, kb + RIB, (b8 - kb - RIB) / 8, warp, lane);
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

// Rows per CTA: the fewest that leave one wave (a 128-column triangle allows
// one CTA per SM, a 64-column one three).
template <bool UNIT, typename TX>
int rlt_any(const double* L, long ld, TX* X, long ldx, int b, long m, const int* guard, int guard_limit,
            cudaStream_t st) {
  if (m <= 0 || b <= 0) return FLA_SUCCESS;
  if (b > RB) {
    set_last_error("triangular solve: triangle wider than 128");
    return FLA_FAILURE;
  }
  const long wave = (long)ctx().num_sms * (b <= 64 ? 3 : 1);
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
