// Reverse-mode differentiation of the Cholesky factorization and of the
// operations a Gaussian-process likelihood builds on it (no counterpart in
// the reference; the forward operations are FLA_Chol,
// src/lapack/dec/chol/front/flamec/FLA_Chol.c:16-29, and FLA_Trsm,
// src/base/flamec/blas/3/trsm/front/flamec/FLA_Trsm.c:15-26).
//
// Cholesky adjoint, blocked, right to left, in place over Lbar (Murray 2016,
// "Differentiation of the Cholesky decomposition", level-3 reverse mode).
// For the block column J (rows/columns j0 .. j0+w) write
//   R = L(J, 0:j0), D = L(J, J), B = L(below, 0:j0), C = L(below, J)
// and the same names with a bar for the adjoints stored in Lbar:
//   Cbar := Cbar inv(D)                         (GEMM with inv(D))
//   Dbar := adjoint of chol(D) at Dbar - tril(Cbar^T C)
//                                                (GEMM, chol_adj_diag_kernel)
//   Rbar := Rbar - (Dbar + Dbar^T) R - Cbar^T B  (one DMMA GEMM)
//   Bbar := Bbar - Cbar R                        (DMMA GEMM)
// On return the lower triangle of Lbar holds Abar, the adjoint of the lower
// entries of A that the forward factorization reads; the gradient with
// respect to a symmetric A is (Abar + Abar^T) / 2.
#include <algorithm>
#include <climits>
#include <cmath>
#include <string>
#include <vector>

#include "common.h"
#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int AB = 128;          // block size

// Adjoint of one diagonal block D = L(J, J) of order w <= 128, from the
// matrix form of the reverse mode (Murray 2016, eq. for the unblocked case):
//   M = tril(D^T Dbar) + tril(D^T Dbar)^T, its diagonal taken once,
//   S = inv(D)^T M inv(D)  (symmetric),
//   Dbar := tril(S) with half its diagonal,   Dbar + Dbar^T = S.
// Bound by the FP64 tensor rate of the SMs it runs on: a cluster of
// ADJ_CL = 8 CTAs, each owning 16 columns.  All four products have the form
// X^T Z with X lower triangular (D, Dbar, inv(D), inv(D)) and Z 128 x 16, so
// X sits in shared memory once per product, k starts at the row tile, and
// the warps take row tiles t and 15 - t to balance the triangle.  M's
// columns need no exchange (column c of M is D^T Dbar(:, c) below the
// diagonal and Dbar^T D(:, c) above it); Y = inv(D)^T M is transposed into
// the owners of its rows through distributed shared memory, and the last
// product uses S = S^T: S(:, J) = inv(D)^T Y(J, :)^T.
// The column-by-column recurrence on one SM that this replaces took 321 us
// per block (128 dependent steps): n = 4096, 32 blocks, 18.4 ms with it and
// 4.64 ms with this kernel and the split products below.
constexpr int ADJ_CL = 8;
constexpr int ADJ_W = AB / ADJ_CL;      // columns per CTA
constexpr int ADJ_THREADS = 256;
constexpr int ADJ_LD = AB + 4;          // = 4 mod 16: conflict-free fragments
constexpr size_t ADJ_SMEM = sizeof(double) * ADJ_LD * (size_t)(AB + 3 * ADJ_W);

// acc(tile, n-tile) += X^T Z over k >= the row tile, for the row tiles warp
// and 15 - warp (8 rows each) and the 16 columns of Z.
__device__ __forceinline__ void adj_xtz(const double* __restrict__ sX, const double* __restrict__ sZ, int warp,
                                        int lane, double (&acc)[2][2][2]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i0 = 8 * (h ? 15 - warp : warp);
#pragma unroll
    for (int q = 0; q < 2; ++q) acc[h][q][0] = acc[h][q][1] = 0.0;
    const double* xa = sX + (i0 + g) * ADJ_LD + t;
    const double* z0 = sZ + g * ADJ_LD + t;
    const double* z1 = z0 + 8 * ADJ_LD;
#pragma unroll 4
    for (int k = i0; k < AB; k += 4) {
      const double a = xa[k], b0 = z0[k], b1 = z1[k];
      dmma_884(acc[h][0][0], acc[h][0][1], a, b0);
      dmma_884(acc[h][1][0], acc[h][1][1], a, b1);
    }
  }
}

// G: the w x w product Cbar^T C that Dbar loses first (ld AB; null: none).
// Sout: S, w x w, ld lds.
__global__ void __cluster_dims__(ADJ_CL, 1, 1) __launch_bounds__(ADJ_THREADS)
    chol_adj_diag_kernel(const double* __restrict__ L, const double* __restrict__ Dinv, double* Lb, long ld, int w,
                         const double* __restrict__ G, double* __restrict__ Sout, long lds) {
  chain_begin();
  extern __shared__ double asm_[];
  double* sX = asm_;                        // lower triangular operand, zero above
  double* sD = sX + AB * ADJ_LD;            // 16 columns of D, later of M
  double* sB = sD + ADJ_W * ADJ_LD;         // 16 columns of Dbar
  double* sY = sB + ADJ_W * ADJ_LD;         // Y(J, :)^T, written by the whole cluster
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x;              // one cluster: the CTA's rank in it
  const int c0 = rank * ADJ_W;
  auto in = [&](int i, int j) { return i >= j && i < w; };
  auto dbar = [&](int i, int j) { return Lb[i + (long)j * ld] - (G ? G[i + j * AB] : 0.0); };
  // 128 x 128 triangle, sixteen loads in flight per thread
  auto load_x = [&](auto val) {
    for (int e0 = tid; e0 < AB * AB; e0 += ADJ_THREADS * 16) {
      double v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int e = e0 + u * ADJ_THREADS, i = e & (AB - 1), j = e >> 7;
        v[u] = in(i, j) ? val(i, j) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int e = e0 + u * ADJ_THREADS;
        sX[(e & (AB - 1)) + (e >> 7) * ADJ_LD] = v[u];
      }
    }
  };
  // triangles that are only copied: asynchronous copies, all in flight, in
  // pairs of rows where the source allows it
  auto copy_x = [&](const double* __restrict__ src, long lds) {
    const bool vec = ((reinterpret_cast<uintptr_t>(src) | (uintptr_t)(lds * 8)) & 15u) == 0;
    for (int e = tid; e < AB * AB / 2; e += ADJ_THREADS) {
      const int i = (e & (AB / 2 - 1)) * 2, j = e >> 6;
      double* d = sX + i + j * ADJ_LD;
      if (vec && i > j && i + 1 < w) {
        cp_async16(d, src + i + (long)j * lds, 16);
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (in(i + u, j))
            cp_async8(d + u, src + i + u + (long)j * lds);
          else d[u] = 0.0;
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  };
  copy_x(L, ld);
  {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = tid + u * ADJ_THREADS, i = e & (AB - 1), j = c0 + (e >> 7);
      v[u] = in(i, j) ? dbar(i, j) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = tid + u * ADJ_THREADS, i = e & (AB - 1), q = e >> 7;
      sB[i + q * ADJ_LD] = v[u];
    }
  }
  __syncthreads();
  for (int e = tid; e < ADJ_W * AB; e += ADJ_THREADS) {
    const int i = e & (AB - 1), q = e >> 7;
    sD[i + q * ADJ_LD] = sX[i + (c0 + q) * ADJ_LD];
  }
  double v1[2][2][2], v2[2][2][2];
  adj_xtz(sX, sB, warp, lane, v1);  // D^T Dbar(:, J)
  __syncthreads();
  load_x(dbar);
  __syncthreads();
  adj_xtz(sX, sD, warp, lane, v2);  // Dbar^T D(:, J)
  __syncthreads();
  copy_x(Dinv, AB);
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = 8 * (h ? 15 - warp : warp) + g;
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * q + 2 * t + e;
        sD[i + c * ADJ_LD] = i >= c0 + c ? v1[h][q][e] : v2[h][q][e];
      }
  }
  // every CTA of the cluster has started (its shared memory may be written)
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  adj_xtz(sX, sD, warp, lane, v1);  // Y(:, J) = inv(D)^T M(:, J)
  const uint32_t ybase = smem_u32(sY);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = 8 * (h ? 15 - warp : warp) + g;
    const uint32_t row = ybase + (uint32_t)((i & (ADJ_W - 1)) * ADJ_LD) * 8u;
    const uint32_t peer = mapa_shared(row, (uint32_t)(i / ADJ_W));
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer + (uint32_t)(c0 + 8 * q + 2 * t + e) * 8u),
                     "d"(v1[h][q][e])
                     : "memory");
  }
  // release / acquire at cluster scope: Y is complete; it is also the last
  // access to a peer's shared memory, so a CTA may exit on its own after it
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  chain_next();
  adj_xtz(sX, sY, warp, lane, v1);  // S(:, J) = inv(D)^T Y(J, :)^T
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = 8 * (h ? 15 - warp : warp) + g;
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + 8 * q + 2 * t + e;
        if (i >= w || c >= w) continue;
        const double s = v1[h][q][e];
        Sout[i + (long)c * lds] = s;
        if (i > c) Lb[i + (long)c * ld] = s;
        else if (i == c) Lb[i + (long)c * ld] = 0.5 * s;
      }
  }
}

// Lbar(i, i) += scale / L(i, i)
__global__ void logdet_adj_kernel(const double* __restrict__ L, double* __restrict__ Lb, long ld, long n,
                                  double scale) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) Lb[i + i * ld] += scale / L[i + i * ld];
}
// partial sums of log L(i, i)
__global__ void logdet_kernel(const double* __restrict__ L, long ld, long n, double* out) {
  __shared__ double red[256];
  double s = 0.0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    s += log(L[i + i * ld]);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(out, red[0]);
}

bool g_adj_attr = false;

}  // namespace

// Scratch of chol_adjoint_dev for order n, in doubles: the inverses of all
// diagonal blocks, two W (ldw x AB each: S over Cbar, of two consecutive
// blocks), the product Cbar^T C, and room for either stream's partial products:
// `splits` slices of an AB-row GEMM, but no more than a split that fills the
// GPU (four 64 x 64 tiles per SM) ever has.
static long adj_ldw(long n) { return (n + AB + 1) & ~1L; }
static size_t adj_split_elems(long n, int splits) {
  return std::min((size_t)splits * AB * (size_t)(n + AB), (size_t)4 * ctx().num_sms * 64 * 64);
}
size_t chol_adjoint_scratch(long n, int splits) {
  const size_t nblk = (size_t)((n + AB - 1) / AB);
  return nblk * AB * AB + 2 * (size_t)adj_ldw(n) * AB + (size_t)AB * AB + 2 * adj_split_elems(n, splits);
}

// In place over Lb (lower triangle); L lower Cholesky factor; n x n, ld.
// scratch: chol_adjoint_scratch(n, splits) doubles of device memory, used by
// this call alone until its work is done.
//
// The chain from block to block (Cbar inv(D), Cbar^T C, the diagonal block,
// and the updates of the next block's columns) runs on `sd`; the updates of
// the columns left of the next block run on `st`, one block behind, beside the
// next block's chain.  sd == st: in stream order (the batched form, whose
// matrices overlap one another).  n = 4096: 4.46 ms in stream order, 3.81
// ms so (3.41 with launch_chain).
int chol_adjoint_dev(const double* L, double* Lb, long ld, long n, cudaStream_t st, cudaStream_t sd, double* scratch,
                     int splits) {
  if (n <= 0) return FLA_SUCCESS;
  if (!g_adj_attr) {
    FB_CK(cudaFuncSetAttribute(chol_adj_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ADJ_SMEM));
    g_adj_attr = true;
  }
  const long nblk = (n + AB - 1) / AB;
  const long ldw = adj_ldw(n);
  double* Dinv = scratch;
  double* W2 = Dinv + (size_t)nblk * AB * AB;
  double* G = W2 + 2 * (size_t)ldw * AB;
  GemmSplit sp_chain, sp_rest;
  sp_chain.p = G + (size_t)AB * AB;
  sp_chain.elems = sp_rest.elems = adj_split_elems(n, splits);
  sp_rest.p = sp_chain.p + sp_chain.elems;
  auto Lat = [&](long i, long j) { return L + i + j * ld; };
  auto Bat = [&](long i, long j) { return Lb + i + j * ld; };
  const bool two = sd != st;
  cudaEvent_t ev_chain = ctx().ev[0], ev_rest = ctx().ev[1];
  if (tri_inverse_blocks(L, ld, n, true, false, Dinv, st) != FLA_SUCCESS) return FLA_FAILURE;
  if (two) {
    FB_CK(cudaEventRecord(ev_rest, st));
    FB_CK(cudaStreamWaitEvent(sd, ev_rest, 0));
  }
  // columns [c0, c1) left of block q lose its contribution (rows j0 .. n - 1):
  //   Rbar := Rbar - (Dbar + Dbar^T) R - Cbar^T B: S over Cbar in W against R
  //   over B, one product of depth w + m;  Bbar := Bbar - Cbar R
  auto update = [&](const double* W, long j0, int w, long m, long c0, long c1, cudaStream_t s,
                    const GemmSplit* sp) -> int {
    if (c1 <= c0) return FLA_SUCCESS;
    if (gemm_f64(s, true, false, w, c1 - c0, w + m, -1.0, W, ldw, Lat(j0, c0), ld, 1.0, Bat(j0, c0), ld, GEMM_FULL, 0,
                 nullptr, 0, 0, sp) != FLA_SUCCESS)
      return FLA_FAILURE;
    if (m > 0 && gemm_f64(s, false, false, m, c1 - c0, w, -1.0, W + w, ldw, Lat(j0, c0), ld, 1.0, Bat(j0 + w, c0), ld) !=
                     FLA_SUCCESS)
      return FLA_FAILURE;
    return FLA_SUCCESS;
  };
  for (long q = nblk - 1; q >= 0; --q) {
    const long j0 = q * AB;
    const int w = (int)std::min<long>(AB, n - j0);
    const long m = n - j0 - w;  // rows below the block (w = AB when there are any)
    const long jn = std::max<long>(0, j0 - AB);  // the next block's first column
    const double* Dq = Dinv + (size_t)q * AB * AB;
    double* W = W2 + (size_t)(q & 1) * ldw * AB;
    double* Cb = W + w;  // Cbar, below the block's S in W
    if (m > 0) {
      // Cbar := Cbar inv(D)
      if (gemm_f64(sd, false, false, m, w, w, 1.0, Bat(j0 + w, j0), ld, Dq, AB, 0.0, Cb, ldw) != FLA_SUCCESS)
        return FLA_FAILURE;
      // G := Cbar^T C, which Dbar loses in the diagonal kernel
      if (gemm_f64(sd, true, false, w, w, m, 1.0, Cb, ldw, Lat(j0 + w, j0), ld, 0.0, G, AB, GEMM_FULL, 0, nullptr, 0,
                   0, &sp_chain) != FLA_SUCCESS)
        return FLA_FAILURE;
    }
    const int ps = prof_begin(sd);
    FB_LAUNCH(launch_chain(chol_adj_diag_kernel, dim3(ADJ_CL), dim3(ADJ_THREADS), ADJ_SMEM, sd,
        Lat(j0, j0), Dq, Bat(j0, j0), ld, w,
                                                               m > 0 ? G : nullptr, W, ldw));
    prof_end(ps, sd, PROF_DIAG, 2.0 * w * (double)w * w / 3.0);
    count_launch();
    FB_CK(cudaGetLastError());
    if (two) {
      // the next block's columns have the other blocks' contributions once the
      // updates of the block before this one are done
      FB_CK(cudaEventRecord(ev_chain, sd));
      FB_CK(cudaStreamWaitEvent(sd, ev_rest, 0));
      FB_CK(cudaStreamWaitEvent(st, ev_chain, 0));
    }
    if (update(W, j0, w, m, jn, j0, sd, &sp_chain) != FLA_SUCCESS || update(W, j0, w, m, 0, jn, st, &sp_rest) != FLA_SUCCESS)
      return FLA_FAILURE;
    if (m > 0)
      FB_CK(cudaMemcpy2DAsync(Bat(j0 + w, j0), sizeof(double) * ld, Cb, sizeof(double) * ldw, sizeof(double) * m, w,
                              cudaMemcpyDeviceToDevice, st));
    if (two) FB_CK(cudaEventRecord(ev_rest, st));
  }
  if (two) {
    FB_CK(cudaEventRecord(ev_chain, sd));
    FB_CK(cudaStreamWaitEvent(st, ev_chain, 0));
  }
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

// Lbar += scale * diag(1 / L_ii): adjoint of scale * sum_i log L_ii.
int logdet_adjoint_dev(const double* L, double* Lb, long ld, long n, double scale, cudaStream_t st) {
  if (n <= 0) return FLA_SUCCESS;
  logdet_adj_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(L, Lb, ld, n, scale);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

int logdet_dev(const double* L, long ld, long n, double* h_out, cudaStream_t st) {
  double* d = (double*)ws_get(WS_IR2, sizeof(double) * 8);
  if (!d) return FLA_FAILURE;
  FB_CK(cudaMemsetAsync(d, 0, sizeof(double), st));
  logdet_kernel<<<(unsigned)std::min<long>(1024, (n + 255) / 256), 256, 0, st>>>(L, ld, n, d);
  count_launch();
  FB_CK(cudaMemcpyAsync(h_out, d, sizeof(double), cudaMemcpyDeviceToHost, st));
  FB_CK(cudaStreamSynchronize(st));
  return FLA_SUCCESS;
}

// Adjoint of X = inv(L) B (L lower, non-unit, n x n; X, B n x k):
//   Bbar := inv(L)^T Xbar (in place over Xbar), Lbar -= tril(Bbar X^T).
int trsm_adjoint_dev(DMat L, DMat X, DMat Xbar, double* Lb, long ldlb, cudaStream_t st) {
  if (trsm_left_dev(L, Xbar, true, true, false, st) != FLA_SUCCESS) return FLA_FAILURE;
  return gemm_f64(st, false, true, L.m, L.m, X.n, -1.0, Xbar.p, Xbar.ld, X.p, X.ld, 1.0, Lb, ldlb, GEMM_LOWER, 0);
}

}  // namespace fb

using namespace fb;

extern "C" {

// No counterpart in the reference.  Adjoint of the lower Cholesky
// factorization A = L L^T (FLA_Chol): L holds the factor, Lbar (same order)
// the adjoint of L in its lower triangle; on return the lower triangle of
// Lbar holds Abar, the adjoint of the lower entries of A (the gradient with
// respect to a symmetric A is (Abar + Abar^T)/2).  Only the lower triangles
// are read or written.  FLA_DOUBLE objects, device or host buffers.
FLA_Error FLA_Chol_adjoint(FLA_Uplo uplo, FLA_Obj L, FLA_Obj Lbar) {
  if (!ctx().initialized) FLA_Init();
  FB_REQUIRE(uplo == FLA_LOWER_TRIANGULAR, "FLA_Chol_adjoint", "only FLA_LOWER_TRIANGULAR is provided");
  FB_REQUIRE(L.base && Lbar.base && L.base->datatype == FLA_DOUBLE && Lbar.base->datatype == FLA_DOUBLE,
             "FLA_Chol_adjoint", "objects must be FLA_DOUBLE");
  FB_REQUIRE(L.m == L.n && Lbar.m == L.m && Lbar.n == L.n, "FLA_Chol_adjoint", "nonconformal objects");
  if (L.m == 0) return FLA_SUCCESS;
  Staged sl, sb;
  if (stage(L, WS_STAGE_A, &sl) != FLA_SUCCESS || stage(Lbar, WS_STAGE_B, &sb) != FLA_SUCCESS) return FLA_FAILURE;
  if (sl.ld != sb.ld) {
    set_last_error("FLA_Chol_adjoint: L and Lbar need the same leading dimension");
    return FLA_FAILURE;
  }
  cudaStream_t st = ctx().stream;
  op_begin(st);
  double* scr = (double*)ws_get(WS_ADJ, sizeof(double) * chol_adjoint_scratch((long)L.m, 16));
  if (!scr) return FLA_FAILURE;
  if (chol_adjoint_dev((const double*)sl.dev, (double*)sb.dev, sl.ld, (long)L.m, st, ctx().side, scr, 16) !=
      FLA_SUCCESS)
    return FLA_FAILURE;
  op_end(st);
  if (unstage(sb) != FLA_SUCCESS || sync_all() != FLA_SUCCESS) return FLA_FAILURE;
  return FLA_SUCCESS;
}

// Lbar += scale * diag(1/L(i,i)), the adjoint of scale * sum_i log L(i,i)
// (log det A = 2 sum_i log L(i,i)); *logdet (optional) receives
// sum_i log L(i,i).
FLA_Error FLA_B200_Chol_logdet_adjoint(FLA_Obj L, FLA_Obj Lbar, double scale, double* logdet) {
  if (!ctx().initialized) FLA_Init();
  FB_REQUIRE(L.base && Lbar.base && L.m == L.n && Lbar.m == L.m && Lbar.n == L.n, "FLA_B200_Chol_logdet_adjoint",
             "nonconformal objects");
  Staged sl, sb;
  if (stage(L, WS_STAGE_A, &sl) != FLA_SUCCESS || stage(Lbar, WS_STAGE_B, &sb) != FLA_SUCCESS) return FLA_FAILURE;
  if (sl.ld != sb.ld) {
    set_last_error("FLA_B200_Chol_logdet_adjoint: L and Lbar need the same leading dimension");
    return FLA_FAILURE;
  }
  cudaStream_t st = ctx().stream;
  op_begin(st);
  if (logdet && logdet_dev((const double*)sl.dev, sl.ld, (long)L.m, logdet, st) != FLA_SUCCESS) return FLA_FAILURE;
  if (logdet_adjoint_dev((const double*)sl.dev, (double*)sb.dev, sb.ld, (long)L.m, scale, st) != FLA_SUCCESS)
    return FLA_FAILURE;
  op_end(st);
  if (unstage(sb) != FLA_SUCCESS || sync_all() != FLA_SUCCESS) return FLA_FAILURE;
  return FLA_SUCCESS;
}

// Adjoint of X = inv(L) B (FLA_Trsm left, lower, no transpose, non-unit):
// given X and Xbar (n x k), Xbar := Bbar = inv(L)^T Xbar and Lbar -=
// tril(Bbar X^T).
FLA_Error FLA_B200_Trsm_llnn_adjoint(FLA_Obj L, FLA_Obj X, FLA_Obj Xbar, FLA_Obj Lbar) {
  if (!ctx().initialized) FLA_Init();
  FB_REQUIRE(L.base && X.base && Xbar.base && Lbar.base && L.m == L.n && X.m == L.m && Xbar.m == L.m &&
                 Xbar.n == X.n && Lbar.m == L.m && Lbar.n == L.n,
             "FLA_B200_Trsm_llnn_adjoint", "nonconformal objects");
  Staged sl, sx, sxb, slb;
  if (stage(L, WS_STAGE_A, &sl) != FLA_SUCCESS || stage(X, WS_STAGE_B, &sx) != FLA_SUCCESS ||
      stage(Xbar, WS_STAGE_X, &sxb) != FLA_SUCCESS || stage(Lbar, WS_FB, &slb) != FLA_SUCCESS)
    return FLA_FAILURE;
  cudaStream_t st = ctx().stream;
  auto dm = [](const Staged& s) {
    DMat d;
    d.p = (double*)s.dev;
    d.ld = s.ld;
    d.m = s.m;
    d.n = s.n;
    return d;
  };
  op_begin(st);
  if (trsm_adjoint_dev(dm(sl), dm(sx), dm(sxb), (double*)slb.dev, slb.ld, st) != FLA_SUCCESS) return FLA_FAILURE;
  op_end(st);
  if (unstage(sxb) != FLA_SUCCESS || unstage(slb) != FLA_SUCCESS || sync_all() != FLA_SUCCESS) return FLA_FAILURE;
  return FLA_SUCCESS;
}

// No counterpart in the reference.  FLA_Chol_adjoint over a batch: for each
// i, L[i] (device, order n[i], leading dimension ld[i]) holds a lower
// Cholesky factor and Lbar[i] (device, same order and leading dimension)
// the adjoint of L[i]; first Lbar[i](j, j) += logdet_scale / L[i](j, j) (the
// adjoint of logdet_scale * sum_j log L(j, j); 0 skips it), then Lbar[i]'s
// lower triangle is replaced by Abar[i] as FLA_Chol_adjoint does.  Each
// matrix runs the blocked adjoint; the matrices, largest first, are spread
// round-robin over a pool of streams with a scratch area each, so the small
// per-block kernels of different matrices overlap.
FLA_Error FLA_Chol_adjoint_batched(int count, const int* n, double** L, const int* ld, double** Lbar,
                                   double logdet_scale) {
  if (!ctx().initialized) FLA_Init();
  long maxn = 0;
  for (int i = 0; i < count; ++i) {
    FB_REQUIRE(n[i] >= 0 && ld[i] >= std::max(1, n[i]), "FLA_Chol_adjoint_batched", "bad order or leading dimension");
    if (n[i] > 0 && (!is_device_ptr(L[i]) || !is_device_ptr(Lbar[i]))) {
      set_last_error("FLA_Chol_adjoint_batched: matrix " + std::to_string(i) + ": buffers must be device memory");
      return FLA_FAILURE;
    }
    maxn = std::max<long>(maxn, n[i]);
  }
  if (count <= 0 || maxn == 0) return FLA_SUCCESS;
  constexpr int NS = 8;
  static cudaStream_t pool[NS];
  static cudaEvent_t ev[NS + 1];
  static bool made = false;
  if (!made) {
    for (int q = 0; q < NS; ++q) FB_CK(cudaStreamCreateWithFlags(&pool[q], cudaStreamNonBlocking));
    for (int q = 0; q <= NS; ++q) FB_CK(cudaEventCreateWithFlags(&ev[q], cudaEventDisableTiming));
    made = true;
  }
  const size_t per = (chol_adjoint_scratch(maxn, 4) + 1) & ~size_t(1);  // keeps each area 16-byte aligned
  double* scr = (double*)ws_get(WS_ADJ, sizeof(double) * per * NS);
  if (!scr) return FLA_FAILURE;
  std::vector<int> order(count);
  for (int i = 0; i < count; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return n[x] > n[y]; });
  cudaStream_t st = ctx().stream;
  op_begin(st);
  FB_CK(cudaEventRecord(ev[NS], st));
  for (int q = 0; q < NS; ++q) FB_CK(cudaStreamWaitEvent(pool[q], ev[NS], 0));
  for (int k = 0; k < count; ++k) {
    const int i = order[k], q = k % NS;
    if (n[i] == 0) continue;
    if (logdet_scale != 0.0 && logdet_adjoint_dev(L[i], Lbar[i], ld[i], n[i], logdet_scale, pool[q]) != FLA_SUCCESS)
      return FLA_FAILURE;
    if (chol_adjoint_dev(L[i], Lbar[i], ld[i], n[i], pool[q], pool[q], scr + per * q, 4) != FLA_SUCCESS) return FLA_FAILURE;
  }
  for (int q = 0; q < NS; ++q) {
    FB_CK(cudaEventRecord(ev[q], pool[q]));
    FB_CK(cudaStreamWaitEvent(st, ev[q], 0));
  }
  op_end(st);
  return sync_all();
}

}  // extern "C"
