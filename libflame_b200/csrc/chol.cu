// FP64 Cholesky factorization (FLA_Chol) on the GPU.
//
// Right-looking blocked algorithm with the reference's structure
// (src/lapack/dec/chol/l/flamec/FLA_Chol_l_blk_var3.c:13-66):
//   for each 128-column block:  A11 := chol(A11)        [potrf_diag_kernel]
//                               A21 := A21 inv(A11)^T   [rlt_kernel, rlt.cu]
//                               A22 -= A21 A21^T (lower) [DMMA GEMM engine]
// with the next block column factored on a second stream while the rest of
// the trailing update runs (chol_lower_enqueue).
// The diagonal block is factored in shared memory in 32-column steps (the
// reference's inner blocksize, FLA_Chol_cntl_init.c:23-61): a warp factors
// each 32x32 block (the unblocked var2/var3 leaf), the rows below are solved
// against it and the trailing part of the block is updated, all in SMEM.
// A failing pivot (<= 0 or NaN, bl1_dsqrte in
// src/base/flamec/blis/include/blis_macro_defs.h:134-136) records the
// zero-based global column in the status block; every later kernel of the
// factorization sees it and returns without touching memory.
#include <algorithm>
#include <climits>
#include <cstdlib>

#include "chol_leaf.cuh"
#include "common.h"
#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int NB = 128;        // outer block
constexpr int IB = CHOL_IB;    // inner block
constexpr int LDS = NB + 4;    // SMEM leading dimension (= 4 mod 16: conflict-free DMMA fragments)
constexpr int POTRF_THREADS = 256;
constexpr int POTRF_SMEM = NB * LDS * 8;
__device__ __forceinline__ bool guard_failed(const int* info) {
  return *((volatile const int*)info) != INT_MAX;
}

// Factor the b x b (b <= 128) lower-triangular diagonal block at A (ld) in
// place.  gcol = global index of its first column for the info word.
// Bound by the pivot chain of one warp: per column a reciprocal square root,
// two products and a shuffle.  Everything else of a 32-column chunk runs
// beside that chain:
//   (a) warp 0 factors the 32 x 32 diagonal block, one row per lane in
//       registers, and publishes each column in shared memory with a counter;
//       warps 1-3 solve the rows below (one row per thread in registers,
//       X := X inv(L11)^T, dtrsm's R,L,T,N order), one column behind warp 0;
//       warps 4-7 subtract the previous chunk's products from the columns
//       beyond this chunk;
//   (b) all warps subtract this chunk's products from the next 32 columns.
// The products run on the FP64 tensor cores.  The pivot chain carries register
// values only: the next pivot is formed by its own lane from its own
// multiplier (fma(-l, l, a)) and shuffled; each pivot's reciprocal square root
// is one rsqrt, its square root d * rsqrt(d).
// Measured (128 x 128): 40 us with the solve and the products between the
// chunks' chains, 27 us in this form.
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// S(r, c) -= sum_{k < IB} S(r, jb + k) S(c, jb + k) for 8 x 8 tiles: rows
// r_lo + 8 i, columns c_lo + 8 j (i < nti, j < ntj), tiles on or below the
// diagonal only (r_lo, c_lo multiples of 8), dealt to the warps w, w + nw, ...
// Entries above the diagonal of a diagonal tile are written too: nothing
// reads them.
__device__ __forceinline__ void syrk_tiles(double* S, int jb, int r_lo, int nti, int c_lo, int ntj, int w, int nw,
                                           int lane) {
  const int g = lane >> 2, t = lane & 3;
  for (int e = w; e < nti * ntj; e += nw) {
    const int r = r_lo + 8 * (e % nti), c = c_lo + 8 * (e / nti);
    if (r < c) continue;
    const double* pa = S + r + g + (jb + t) * LDS;
    const double* pb = S + c + g + (jb + t) * LDS;
    double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < IB; k += 8) {
      dmma_884(d0[0], d0[1], pa[k * LDS], pb[k * LDS]);
      dmma_884(d1[0], d1[1], pa[(k + 4) * LDS], pb[(k + 4) * LDS]);
    }
    double* o = S + r + g + (c + 2 * t) * LDS;
    o[0] -= d0[0] + d1[0];
    o[LDS] -= d0[1] + d1[1];
  }
}

__global__ void __launch_bounds__(POTRF_THREADS, 1) potrf_diag_kernel(double* A, long ld, int b, int gcol,
                                                                   int* info, int* err) {
  chain_begin();
  extern __shared__ __align__(16) double S[];  // S[r + c*LDS]
  __shared__ int s_fail, s_cnt;
  __shared__ double s_rinv[2][IB];
  if (guard_failed(info)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // load the lower triangle (and diagonal) with asynchronous copies, all in
  // flight at once; the rest of the square only feeds entries nobody reads
  for (int c = warp; c < b; c += POTRF_THREADS / 32)
    for (int r = c + lane; r < b; r += 32) cp_async8(S + r + c * LDS, A + r + (long)c * ld);
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (tid == 0) {
    s_fail = -1;
    s_cnt = 0;
  }
  __syncthreads();
  const int b8 = (b + 7) & ~7;
  for (int jb = 0; jb < b; jb += IB) {
    const int w = min(IB, b - jb), r0 = jb + w;  // r0: first row below the block
    // (a); the counter runs on over the chunks (base jb), s_rinv alternates
    double* rinv = s_rinv[(jb / IB) & 1];
    if (warp == 0) {
      potrf_diag32<LDS>(S, jb, w, lane, rinv, &s_cnt, jb, &s_fail);
    } else if (warp < 4) {
      const int r = r0 + (warp - 1) * 32 + lane;
      if (r < b) potrf_row<LDS>(S, jb, r, rinv, &s_cnt, jb, err);
    } else if (jb > 0 && r0 < b) {
      syrk_tiles(S, jb - IB, r0, (b8 - r0) / 8, r0, (b8 - r0) / 8, warp - 4, 4, lane);
    }
    __syncthreads();
    if (s_fail >= 0) break;
    // (b) the next chunk's columns
    if (r0 < b) syrk_tiles(S, jb, r0, (b8 - r0) / 8, r0, min(IB, b8 - r0) / 8, warp, POTRF_THREADS / 32, lane);
    __syncthreads();
  }
  chain_next();
  // write back the lower triangle (the strictly upper part of A is untouched)
  for (int c = warp; c < b; c += POTRF_THREADS / 32)
    for (int r = c + lane; r < b; r += 32) A[r + (long)c * ld] = S[r + c * LDS];
  if (tid == 0 && s_fail >= 0) atomicMin(info, gcol + s_fail);
}

bool g_attr_done = false;
void set_attrs() {
  if (g_attr_done) return;
  cudaFuncSetAttribute(potrf_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, POTRF_SMEM);
  g_attr_done = true;
}

}  // namespace

// Outer blocksize of FLA_Chol: the depth of the trailing updates.  256 by
// default (the DMMA GEMM runs its K=256 updates about a fifth faster than
// K=128 ones); FLA_B200_CHOL_BLOCKSIZE = 128 or 256 overrides it.
int chol_blocksize() {
  static int nb = 0;
  if (nb == 0) {
    nb = 256;
    if (const char* e = std::getenv("FLA_B200_CHOL_BLOCKSIZE")) {
      const int v = std::atoi(e);
      if (v == 128 || v == 256) nb = v;
    }
  }
  return nb;
}

// Enqueue the blocked factorization of the lower triangle of A on `st`.
// Outer blocks of NBO = 128 or 256 columns; each outer panel is factored as
// 128-column sub-panels:
//   sub-panel j:   A11 := chol(A11);
//                  A21 := A21 inv(L11)^T in one launch;
//                  the panel's later columns -= A21 A21^T
//   then the panel's rows below its diagonal block are copied transposed,
//   and step k updates A22(:, next panel) -= A21 A21(next rows)^T, factors
//   the next panel on the second stream, and meanwhile updates
//   A22(rest) -= A21 A21^T (lower) on the main stream.
// Failure semantics follow FLA_Chol_l_blk_var3: the updates of step k run
// unless a column before k + b has failed (the guard limit of each launch),
// so a failure in the next panel does not cut short step k's update.
int chol_lower_enqueue(DMat A, cudaStream_t st) {
  set_attrs();
  Context& cx = ctx();
  const long n = A.m, ld = A.ld;
  if (n <= 0) return FLA_SUCCESS;
  int* info = cx.d_status + ST_INFO;
  // The next panel is factored on the library's second stream beside the
  // trailing update (as in FLA_LU_piv); FLA_B200_CHOL_LOOKAHEAD=0 keeps the
  // panels in stream order.  Only calls on the library's main stream
  // overlap; a call on another stream runs in that stream's order.
  static const bool look = [] {
    const char* e = std::getenv("FLA_B200_CHOL_LOOKAHEAD");
    return !(e && e[0] == '0');
  }();
  cudaStream_t sd = (look && st == cx.stream) ? cx.side : st;
  const long NBO = chol_blocksize();
  // Transposed copy of each factored outer panel's rows below its diagonal
  // block (NBO x rows, k contiguous), two buffers used in turn: the
  // lookahead and trailing updates take their second operand from it
  // k-contiguous (one 16 x 64 TMA box per stage, the LU's operand shape).
  const long ldpt = NBO;
  double* PT = (double*)ws_get(WS_PANEL_T, sizeof(double) * 2 * (size_t)ldpt * (size_t)std::max<long>(n, 1));
  if (!PT) return FLA_FAILURE;
  auto pt_of = [&](long k) { return PT + ((k / NBO) & 1) * (size_t)ldpt * (size_t)n; };
  cudaEvent_t ev_look = cx.ev[2], ev_panel = cx.ev[3];
  auto at = [&](long i, long j) { return A.p + i + j * ld; };

  // 128-column sub-panel at column k: diagonal block and the block column
  // below it.
  auto sub = [&](long k, cudaStream_t s) -> int {
    const int b = (int)std::min<long>(NB, n - k);
    int ps = prof_begin(s);
    FB_LAUNCH(launch_chain(potrf_diag_kernel, dim3(1), dim3(POTRF_THREADS), POTRF_SMEM, s,
        at(k, k), ld, b, (int)k, info, cx.d_status + ST_ERROR));
    prof_end(ps, s, PROF_DIAG, (double)b * b * b / 3.0);
    count_launch();
    FB_CK(cudaGetLastError());
    const long m2 = n - k - b;
    if (m2 <= 0) return FLA_SUCCESS;
    return trsm_rlt_subst(at(k, k), at(k + b, k), ld, b, m2, info, (int)(k + b), s);
  };
  // Outer panel at column k: its sub-panels left to right, each followed by
  // the update of the panel's remaining columns; then the transposed copy of
  // its rows below the diagonal block.
  auto panel = [&](long k, cudaStream_t s) -> int {
    const long kend = std::min<long>(n, k + NBO);
    for (long j = k; j < kend; j += NB) {
      if (sub(j, s) != FLA_SUCCESS) return FLA_FAILURE;
      const long bj = std::min<long>(NB, n - j), j2 = j + bj;
      if (j2 >= kend) break;
      if (gemm_f64(s, false, true, n - j2, kend - j2, bj, -1.0, at(j2, j), ld, at(j2, j), ld, 1.0, at(j2, j2), ld,
                   GEMM_LOWER, 0, info, (int)j2) != FLA_SUCCESS)
        return FLA_FAILURE;
    }
    if (n > kend)
      return transpose_dev(at(kend, k), ld, pt_of(k), ldpt, n - kend, kend - k, false, s);
    return FLA_SUCCESS;
  };

  if (panel(0, st) != FLA_SUCCESS) return FLA_FAILURE;
  for (long k = 0; k < n; k += NBO) {
    const long b = std::min<long>(NBO, n - k);
    const long m2 = n - k - b;
    if (m2 <= 0) break;
    const int lim = (int)(k + b);
    const long nb2 = std::min<long>(NBO, m2);
    // the next panel's columns first; op(B) = panel^T from its transposed copy
    // (column c of the copy is panel row k + b + c)
    const double* pt = pt_of(k);
    if (gemm_f64(st, false, false, m2, nb2, b, -1.0, at(k + b, k), ld, pt, ldpt, 1.0, at(k + b, k + b), ld,
                 GEMM_LOWER, 0, info, lim) != FLA_SUCCESS)
      return FLA_FAILURE;
    FB_CK(cudaEventRecord(ev_look, st));
    FB_CK(cudaStreamWaitEvent(sd, ev_look, 0));
    if (panel(k + b, sd) != FLA_SUCCESS) return FLA_FAILURE;
    FB_CK(cudaEventRecord(ev_panel, sd));
    if (m2 > nb2 &&
        gemm_f64(st, false, false, m2 - nb2, m2 - nb2, b, -1.0, at(k + b + nb2, k), ld, pt + nb2 * ldpt, ldpt, 1.0,
                 at(k + b + nb2, k + b + nb2), ld, GEMM_LOWER, 0, info, lim) != FLA_SUCCESS)
      return FLA_FAILURE;
    FB_CK(cudaStreamWaitEvent(st, ev_panel, 0));
  }
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

// Factor one b x b (b <= 128) lower diagonal block in place (FP64); gcol is
// the global index of its first column for the info word.
int potrf_diag_dev(double* A, long ld, int b, int gcol, cudaStream_t st) {
  set_attrs();
  int ps = prof_begin(st);
  FB_LAUNCH(launch_chain(potrf_diag_kernel, dim3(1), dim3(POTRF_THREADS), POTRF_SMEM, st,
        A, ld, b, gcol, ctx().d_status + ST_INFO,
                                                            ctx().d_status + ST_ERROR));
  prof_end(ps, st, PROF_DIAG, (double)b * b * b / 3.0);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

int chol_lower_dev(DMat A, int* info) {
  if (A.m == 0) {
    *info = -1;
    return FLA_SUCCESS;
  }
  if (status_reset() != FLA_SUCCESS) return FLA_FAILURE;
  if (chol_lower_enqueue(A, ctx().stream) != FLA_SUCCESS) return FLA_FAILURE;
  return status_read(info);
}

}  // namespace fb
