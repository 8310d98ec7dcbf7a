// Application of Q from its UT representation to a block of columns
// (FLA_Apply_Q_UT), B200 form.
//
// Reference: FLA_Apply_Q_UT_lhfc_blk_var1.c:148-182 (src/lapack/util/app/qut/
// lhfc/flamec), block by block: W := T^-T (U^T B), B -= U W.
//
// The blocks are grouped into super-blocks of s <= 128 columns (a multiple of
// b_alg).  What does not depend on B is formed for all super-blocks at once:
// the Gram blocks U_i^T U_j that complete each super-block's triangular
// factor (qr_gram_kernel), the factors (qr_assemble_kernel) and their
// inverses (one launch).  Then each super-block takes three launches, in
// order:
//   P_z  := slices of U2^T B2             (DMMA GEMM, slices left unadded)
//   W2   := Ti^T (sum P_z + U1^T B1), B1 -= U1 W2     (qr_apply_mid_kernel)
//   B2   -= U2 W2                          (DMMA GEMM)
// with U = [U1; U2], U1 the s x s unit lower triangle at its top: the GEMMs
// read the stored reflectors in place and only the small kernel knows about
// the triangle (no copy of U with explicit ones and zeros).
// Bound by the latency of that chain; before, each super-block had copies of
// U and B, a Gram product with a 4-tile output, an inverse on one SM and a
// reduction in it: m = 8192, k = 4096, 64 columns 2.88 ms,
// now 1.38 ms (three launches of 8 to 16 us per super-block, 0.3 ms before
// them).
#include <algorithm>

#include "common.h"
#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int AS = 128;           // widest super-block
constexpr int ALD = AS + 4;       // = 4 mod 16: conflict-free fragments
constexpr int GK = 64;            // rows of a Gram slab
constexpr int GLD = GK + 4;
constexpr size_t GRAM_SMEM = sizeof(double) * AS * GLD;
constexpr int MID_THREADS = 512;
constexpr int MID_COLS = 8;
constexpr size_t MID_SMEM = sizeof(double) * ((size_t)AS * ALD + 3 * MID_COLS * ALD);

// Partial Gram matrices: slice z = blockIdx.x of super-block q = blockIdx.y
// adds U(rows, :)^T U(rows, :) over the slabs z, z + gridDim.x, ... of GK
// rows of its trapezoid (unit diagonal, zeros above) and writes the tiles on
// and above the diagonal to P + (q gridDim.x + z) AS^2 (ld AS).  Bound by the
// FP64 tensor rate (s^2 (m - jb) flops a super-block).  A warp owns the tile
// rows w and 15 - w: 17 of the 136 upper 8 x 8 tiles for every warp.
__global__ void __launch_bounds__(256) qr_gram_kernel(const double* __restrict__ U, long ldu, long m, int k, int S,
                                                      double* __restrict__ P) {
  extern __shared__ __align__(16) double gram_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const long jb = (long)blockIdx.y * S;
  const int s = (int)(k - jb < S ? k - jb : S);
  const long M = m - jb;
  const double* Uq = U + jb + jb * ldu;
  double a0[16][2], a1[8][2];
#pragma unroll
  for (int j = 0; j < 16; ++j) a0[j][0] = a0[j][1] = 0.0;
#pragma unroll
  for (int j = 0; j < 8; ++j) a1[j][0] = a1[j][1] = 0.0;
  for (long r0 = (long)blockIdx.x * GK; r0 < M; r0 += (long)gridDim.x * GK) {
    __syncthreads();
#pragma unroll 8
    for (int e = tid; e < GK * AS; e += 256) {
      const int r = e % GK, c = e / GK;
      const long i = r0 + r;
      double* d = gram_sm + r + c * GLD;
      if (i < M && c < s && i > c) cp_async8(d, Uq + i + (long)c * ldu);
      else *d = (i == c && c < s) ? 1.0 : 0.0;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const double* p = gram_sm + t + g * GLD;
#pragma unroll 1
    for (int kk = 0; kk < GK; kk += 4) {
      const double x0 = p[kk + 8 * warp * GLD], x1 = p[kk + 8 * (15 - warp) * GLD];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j >= warp) {
          const double b = p[kk + 8 * j * GLD];
          dmma_884(a0[j][0], a0[j][1], x0, b);
          if (j >= 8 && j >= 15 - warp) dmma_884(a1[j - 8 < 0 ? 0 : j - 8][0], a1[j - 8 < 0 ? 0 : j - 8][1], x1, b);
        }
    }
  }
  double* out = P + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * AS * AS;
#pragma unroll
  for (int j = 0; j < 16; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = 8 * j + 2 * t + e;
      if (j >= warp) out[8 * warp + g + c * AS] = a0[j][e];
      if (j >= 8 && j >= 15 - warp) out[8 * (15 - warp) + g + c * AS] = a1[j - 8 < 0 ? 0 : j - 8][e];
    }
}

// Triangular factor of super-block q = blockIdx.y (order s, ld S) at Ts + q S
// (S + 1): the stored b_alg x b_alg T blocks on its diagonal, the Gram blocks
// (nz slices added in order) above them.  The spacing is that of diagonal
// blocks of a matrix with leading dimension S, as the batched inverse takes
// them.
__global__ void __launch_bounds__(256) qr_assemble_kernel(const double* __restrict__ T, long ldt, int b_alg, int k,
                                                          int S, const double* __restrict__ P, int nz,
                                                          double* __restrict__ Ts) {
  const int q = blockIdx.y;
  const long jb = (long)q * S;
  const int s = (int)(k - jb < S ? k - jb : S);
  const double* Pq = P + (size_t)q * nz * AS * AS;
  double* out = Ts + (size_t)q * S * (S + 1);
  for (int e = blockIdx.x * 256 + threadIdx.x; e < s * s; e += gridDim.x * 256) {
    const int i = e % s, j = e / s;
    if (i > j) continue;
    double v = 0.0;
    if (i / b_alg == j / b_alg) {
      v = T[(i % b_alg) + (jb + j) * ldt];
    } else {
#pragma unroll 4
      for (int z = 0; z < nz; ++z) v += Pq[(size_t)z * AS * AS + i + j * AS];
    }
    out[i + (long)j * S] = v;
  }
}

// acc += sum_k a(k) Z(k, 0..7) over k in [k_lo, k_hi) (multiples of 4), two
// accumulator chains.
template <class LoadA>
__device__ __forceinline__ void mid_product(LoadA a, const double* z, int k_lo, int k_hi, double (&r)[2]) {
  double c[2][2] = {};
  int k = k_lo;
  for (; k + 4 < k_hi; k += 8) {
    dmma_884(c[0][0], c[0][1], a(k), z[k]);
    dmma_884(c[1][0], c[1][1], a(k + 4), z[k + 4]);
  }
  if (k < k_hi) dmma_884(c[0][0], c[0][1], a(k), z[k]);
  r[0] = c[0][0] + c[1][0];
  r[1] = c[0][1] + c[1][1];
}

// For MID_COLS columns of B: W := sum_z P_z + U1^T B1, W2 := Ti^T W
// (transpose) or Ti W, B1 -= U1 W2.  U1 has h = s rows, or s + 1 when s is
// odd and there is one more (so that U2 and B2 start on 16 bytes).  P_z: s x nr slices (ld ldp, zs apart,
// nz of them).  U1 (strictly lower, implicit ones) and Ti (upper) share one
// square of shared memory; a warp owns one 8-row tile of each product.
__global__ void __launch_bounds__(MID_THREADS) qr_apply_mid_kernel(const double* __restrict__ U1, long ldu,
                                                                   const double* __restrict__ Ti, long ldti, int s, int h,
                                                                   const double* __restrict__ P, long ldp, long zs,
                                                                   int nz, int transpose, double* B, long ldb, int nr,
                                                                   double* __restrict__ W2, long ldw) {
  chain_begin();
  extern __shared__ __align__(16) double mid_sm[];
  double* sQ = mid_sm;                       // U1(i, j), i > j;  Ti(i, j), i <= j
  double* sB = sQ + AS * ALD;                // B1 columns
  double* sW = sB + MID_COLS * ALD;          // W
  double* sV = sW + MID_COLS * ALD;          // W2
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int c0 = blockIdx.x * MID_COLS, nc = min(MID_COLS, nr - c0);
#pragma unroll 8
  for (int e = tid; e < AS * AS; e += MID_THREADS) {
    const int i = e & (AS - 1), j = e >> 7;
    double* d = sQ + i + j * ALD;
    if (i < h && j < s) cp_async8(d, i > j ? U1 + i + (long)j * ldu : Ti + i + (long)j * ldti);
    else *d = 0.0;
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
  for (int u = 0; u < AS * MID_COLS / MID_THREADS; ++u) {
    const int e = tid + u * MID_THREADS, i = e & (AS - 1), c = e >> 7;
    double w = 0.0, b = 0.0;
    if (i < h && c < nc) b = B[i + (long)(c0 + c) * ldb];
    if (i < s && c < nc) {
      const double* p = P + i + (long)(c0 + c) * ldp;
#pragma unroll 16
      for (int z = 0; z < nz; ++z) w += p[(long)z * zs];
    }
    sB[i + c * ALD] = b;
    sW[i + c * ALD] = w;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int i0 = 8 * warp, i = i0 + g;
  const double* zb = sB + t + g * ALD;
  const double* zw = sW + t + g * ALD;
  const double* zv = sV + t + g * ALD;
  const double one = i < s ? 1.0 : 0.0;
  double r[2];
  // U1^T B1: (U1^T)(i, k) = U1(k, i), k > i, one at k = i
  mid_product([&](int k) { const int kk = k + t; return kk > i ? sQ[kk + i * ALD] : kk == i ? one : 0.0; }, zb, i0, AS,
              r);
#pragma unroll
  for (int e = 0; e < 2; ++e) r[e] += sW[i + (2 * t + e) * ALD];
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 2; ++e) sW[i + (2 * t + e) * ALD] = r[e];
  __syncthreads();
  if (transpose)  // Ti^T: Ti(k, i), k <= i
    mid_product([&](int k) { const int kk = k + t; return kk <= i ? sQ[kk + i * ALD] : 0.0; }, zw, 0, i0 + 8, r);
  else            // Ti(i, k), k >= i
    mid_product([&](int k) { const int kk = k + t; return kk >= i ? sQ[i + kk * ALD] : 0.0; }, zw, i0, AS, r);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int c = 2 * t + e;
    sV[i + c * ALD] = r[e];
    if (i < s && c < nc) W2[i + (long)(c0 + c) * ldw] = r[e];
  }
  __syncthreads();
  chain_next();
  // U1 W2: U1(i, k), k < i, one at k = i
  mid_product([&](int k) { const int kk = k + t; return kk < i ? sQ[i + kk * ALD] : kk == i ? one : 0.0; }, zv, 0,
              i0 + 8, r);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int c = 2 * t + e;
    if (i < h && c < nc) B[i + (long)(c0 + c) * ldb] = sB[i + c * ALD] - r[e];
  }
}

}  // namespace

// Super-block width of apply_q_blocks for T blocks of b_alg columns: the
// largest even multiple of b_alg that fits (even: the tiles of U2 and B2
// start on 16-byte boundaries), 0 if there is none.
int apply_q_width(int b_alg) {
  const int u = b_alg % 2 ? 2 * b_alg : b_alg;
  return AS / u * u;
}

// B := Q^T B (transpose_q) or Q B; U (m x k used), B 16-byte aligned with even
// leading dimensions, S = apply_q_width(b_alg) > 0.
int apply_q_blocks(DMat U, long k, DMat T, int b_alg, int S, DMat B, bool transpose_q, cudaStream_t st) {
  const long m = U.m, nr = B.n;
  const long nsb = (k + S - 1) / S;
  const int sms = ctx().num_sms;
  // Gram slices per super-block: about two CTAs per SM over all of them, no
  // more than slabs
  const int nz = (int)std::max<long>(1, std::min<long>(std::min<long>(2L * sms / nsb, 16), (m + GK - 1) / GK));
  // Slices of U2^T B2: no more than the split fills the GPU with (four 64-column
  // tiles per SM), and at most 32: the small kernel adds them
  const long max_slices = std::max<long>(1, std::min<long>(32, 4L * sms / (((S + 127) / 128) * ((nr + 63) / 64))));
  const long ldw = (S + 1) & ~1L;
  const size_t n_gram = (size_t)nsb * nz * AS * AS, n_t = (size_t)nsb * S * (S + 1);
  const size_t n_p = (size_t)max_slices * ldw * nr;
  double* ws = (double*)ws_get(WS_QR_W, sizeof(double) * (std::max(n_gram, n_p) + n_t + (size_t)nsb * S * S +
                                                          (size_t)ldw * nr + 8));
  if (!ws) return FLA_FAILURE;
  double* P = ws;  // Gram slices, then the slices of U2^T B2
  double* Ts = P + std::max(n_gram, n_p);
  double* Ti = Ts + ((n_t + 1) & ~size_t(1));
  double* W2 = Ti + (((size_t)nsb * S * S + 1) & ~size_t(1));
  static bool attr = false;
  if (!attr) {
    FB_CK(cudaFuncSetAttribute(qr_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GRAM_SMEM));
    FB_CK(cudaFuncSetAttribute(qr_apply_mid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MID_SMEM));
    attr = true;
  }
  int ps = prof_begin(st);
  if (S > b_alg) {
    qr_gram_kernel<<<dim3((unsigned)nz, (unsigned)nsb), 256, GRAM_SMEM, st>>>(U.p, U.ld, m, (int)k, S, P);
    count_launch();
  }
  qr_assemble_kernel<<<dim3(8, (unsigned)nsb), 256, 0, st>>>(T.p, T.ld, b_alg, (int)k, S, P, nz, Ts);
  prof_end(ps, st, PROF_OTHER, 0.0);
  count_launch();
  FB_CK(cudaGetLastError());
  if (tri_inverse_blocks_bs(Ts, S, k, S, false, false, Ti, st) != FLA_SUCCESS) return FLA_FAILURE;
  for (long bi = 0; bi < nsb; ++bi) {
    const long q = transpose_q ? bi : nsb - 1 - bi, jb = q * S;
    const int s = (int)std::min<long>(S, k - jb);
    const int h = (int)std::min<long>(m - jb, (s + 1) & ~1);
    const long M2 = m - jb - h;
    const double* Uq = U.p + jb + jb * U.ld;
    double* Bq = B.p + jb;
    GemmSplit sp;
    long slices = 0;
    if (M2 > 0) {
      sp.p = P;
      sp.elems = n_p;
      sp.max_slices = max_slices;
      sp.slices = &slices;
      if (gemm_f64(st, true, false, s, nr, M2, 1.0, Uq + h, U.ld, Bq + h, B.ld, 0.0, nullptr, 0, GEMM_FULL, 0, nullptr,
                   0, 0, &sp) != FLA_SUCCESS)
        return FLA_FAILURE;
    }
    ps = prof_begin(st);
    const long ldp = (s + 1) & ~1L;
    FB_LAUNCH(launch_chain(qr_apply_mid_kernel, dim3((unsigned)((nr + MID_COLS - 1) / MID_COLS)), dim3(MID_THREADS), MID_SMEM, st,
        Uq, U.ld, Ti + (size_t)q * S * S, S, s, h, P, ldp, ldp * nr, (int)slices, transpose_q ? 1 : 0, Bq, B.ld, (int)nr,
        W2, ldw));
    prof_end(ps, st, PROF_TRSM, 3.0 * s * (double)s * nr);
    count_launch();
    FB_CK(cudaGetLastError());
    if (M2 > 0 && gemm_f64(st, false, false, M2, nr, s, -1.0, Uq + h, U.ld, W2, ldw, 1.0, Bq + h, B.ld) != FLA_SUCCESS)
      return FLA_FAILURE;
  }
  return FLA_SUCCESS;
}

}  // namespace fb
