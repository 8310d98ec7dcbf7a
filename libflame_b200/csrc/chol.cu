// FP64 Cholesky factorization (FLA_Chol) on the GPU.
//
// Right-looking blocked algorithm with the reference's structure
// (src/lapack/dec/chol/l/flamec/FLA_Chol_l_blk_var3.c:13-66):
//   for each 128-column block:  A11 := chol(A11)        [potrf_diag_kernel]
//                               A21 := A21 inv(A11)^T   [rlt_kernel, rlt.cu]
//                               A22 -= A21 A21^T (lower) [DMMA GEMM engine]
// with the next block column factored on a second stream while the rest of
// the trailing update runs (chol_lower_enqueue).
// The diagonal block is factored in shared memory in 8-column steps (the
// reference's inner blocksize is 32, FLA_Chol_cntl_init.c:23-61): an 8 x 8
// factor in registers, the rows below solved against it, the products with the
// columns beyond.
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
constexpr int LDS = POTRF_LD;  // SMEM leading dimension
constexpr int POTRF_SMEM = NB * LDS * 8;

__device__ __forceinline__ bool guard_failed(const int* info) {
  return *((volatile const int*)info) != INT_MAX;
}

// Factor the b x b (b <= 128) lower-triangular diagonal block at A (ld) in
// place.  gcol = global index of its first column for the info word.
// Bound by the pivot chain, so as little as possible hangs on it.  Steps of
// eight columns; threads 0..127 own one row each:
//   (a) every warp with rows reads the 8 x 8 diagonal block and factors it
//       redundantly in registers (chol8: no exchange inside the chain, per
//       column a reciprocal square root, a product and a fused multiply-add),
//       then solves its own rows against it (dtrsm's R,L,T,N order); rows of
//       the block itself come out of the same formulas, and the warp that owns
//       them stores them once the other warps have announced (bar.arrive) that
//       they have factored the block, every entry read and used;
//       meanwhile the other warps subtract the previous step's products from the
//       columns beyond this step on the FP64 tensor cores;
//   (b) the rows lose this step's products in the next step's eight columns.
// Measured, one call of FLA_Chol between events (about 6 us without a kernel):
// n = 100 30.7 -> 26.2 us, n = 128 32.2 -> 30.6 us against 32-column blocks
// factored by one warp (lane = row, the column through shared memory, about
// 370 cycles a column); with four instead of twelve warps for the products
// n = 128 took 32.4 us.  With the block's rows stored after the CTA barrier
// instead of the arrivals, n = 1024 (eight blocks) took 336 us, 330 so (324 to
// 328 with the arrivals right after the loads).
__global__ void __launch_bounds__(POTRF_THREADS, 1) potrf_diag_kernel(double* A, long ld, int b, int gcol,
                                                                   int* info) {
  chain_begin();
  extern __shared__ __align__(16) double S[];  // S[r + c*LDS]
  __shared__ int s_fail[2];
  if (guard_failed(info)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // load the lower triangle (and diagonal) with asynchronous copies, all in
  // flight at once; the rest of the square only feeds entries nobody reads
  for (int c = warp; c < b; c += POTRF_THREADS / 32)
    for (int r = c + lane; r < b; r += 32) cp_async8(S + r + c * LDS, A + r + (long)c * ld);
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (tid < 2) s_fail[tid] = -1;
  __syncthreads();
  const int fail = potrf_block(S, b, s_fail);
  chain_next();
  // write back the lower triangle (the strictly upper part of A is untouched)
  for (int c = warp; c < b; c += POTRF_THREADS / 32)
    for (int r = c + lane; r < b; r += 32) A[r + (long)c * ld] = S[r + c * LDS];
  if (tid == 0 && fail >= 0) atomicMin(info, gcol + fail);
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
        at(k, k), ld, b, (int)k, info));
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
        A, ld, b, gcol, ctx().d_status + ST_INFO));
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
