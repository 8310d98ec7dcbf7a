// Batched FP64 LU with partial pivoting (+ solves) for many small matrices of
// uneven sizes (n <= 512): one CTA per matrix, matrices from an atomic counter
// in a host-chosen order (largest first).
//
// Semantics of FLA_LU_piv per matrix (src/lapack/dec/lu/piv/front/flamec/
// FLA_LU_piv.c:16-33): the largest magnitude, the first row among equals; a
// zero pivot column is neither exchanged nor scaled, the first is reported;
// relative pivots.
//
// Right-looking in panels of 32 columns on a row-major copy of [A | B] in the
// CTA's own workspace (the copies of all CTAs fit in L2 up to order 200 with two
// CTAs per SM, from 257 to 310 with one; at order 512 they are 325 MB):
//   panel      rows j..n in registers, one row per thread (lu_leaf.cuh): per
//              column two CTA barriers and an update without memory traffic;
//   exchanges  the composition of the panel's interchanges moves whole rows
//              of the other columns (contiguous) through shared memory;
//   U rows     a thread per column solves with the 32 x 32 unit triangle;
//   update     A22 -= L21 U12 on the FP64 tensor cores (16 x 32 warp tiles,
//              L21 and a chunk of U12 in shared memory).
// The right-hand sides are columns of the copy, so the forward substitution
// and the row exchanges come with the factorization; the backward one follows.
// Bound by the latency of the panels' columns (1 us each at order 512) and, for
// the large orders, the copies' traffic: 148 matrices of order 512 move 5.4 GB
// through HBM (0.6 GB in and out would do; 52 % of the accesses hit L2), 2.5 ms
// at 27 % of its bandwidth.  Orders up to 256 run in CTAs of 256 threads, two per SM, so that one
// matrix's panel overlaps the other's updates; larger ones in CTAs of 512.
// Measured: 2500 matrices, n uniform in 8..512, 4 right-hand sides: 47.4 ms
// with a left-looking panel in shared memory on FP64 FMAs (ten barriers and a
// serial exchange loop per column), 15.0 ms in this form.  (Registers that
// rotate so that one loop body serves every column of the panel were slower:
// 1.1 against 0.96 us a column.)
#include <algorithm>

#include "batched.h"
#include "common.h"
#include "lu_leaf.cuh"

namespace fb {

namespace {

constexpr int LW = 32;            // panel width
constexpr int LSL = LW + 4;       // ld of L21 in shared memory: = 4 mod 16, conflict-free fragments
constexpr int LMAXRHS = 8;        // columns kept for right-hand sides

template <int NT>
struct LuB {
  static constexpr int NW = NT / 32;
  static constexpr int CW = NT / 2;        // columns of U12 per chunk
  static constexpr int LDU = CW + 4;       // = 4 mod 16
  static constexpr int BIG = NT * LSL + LW * LDU;  // L21 and U12; also exchange and transposition buffers
  static constexpr size_t SMEM = sizeof(double) * (BIG + 2 * 2 * LW + LMAXRHS * LW) + 2 * NW * sizeof(RHdr);
  static constexpr int MINB = NT == 256 ? 2 : 1;
};
// workspace of a CTA: rows padded to the update's tiles, columns to 32 plus
// the right-hand sides
__host__ __device__ inline int lub_n32(int n) { return (n + LW - 1) / LW * LW; }
__host__ __device__ inline size_t lub_ws(int n) { return (size_t)(n + 16) * (lub_n32(n) + LMAXRHS); }

// dst(r, c) (row-major, ld ldd) := src(r, c) (column-major, ld lds), nr x nc,
// or the other way round, through one 32 x 33 tile per warp.
template <int NT, bool IN>
__device__ void lub_transpose(double* W, int ldw, double* G, long ldg, int nr, int nc, double* buf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* tile = buf + warp * 32 * 33;
  const int tr = (nr + 31) / 32, tc = (nc + 31) / 32;
  for (int e = warp; e < tr * tc; e += NT / 32) {
    const int r0 = (e % tr) * 32, c0 = (e / tr) * 32;
    double v[32];  // the whole tile in flight
    if (IN) {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        v[q] = (r0 + lane < nr && c0 + q < nc) ? G[(long)(r0 + lane) + (long)(c0 + q) * ldg] : 0.0;
#pragma unroll
      for (int q = 0; q < 32; ++q) tile[lane * 33 + q] = v[q];
      __syncwarp();
#pragma unroll 16
      for (int q = 0; q < 32; ++q)
        if (r0 + q < nr && c0 + lane < nc) W[(long)(r0 + q) * ldw + c0 + lane] = tile[q * 33 + lane];
    } else {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        v[q] = (r0 + q < nr && c0 + lane < nc) ? W[(long)(r0 + q) * ldw + c0 + lane] : 0.0;
#pragma unroll
      for (int q = 0; q < 32; ++q) tile[q * 33 + lane] = v[q];
      __syncwarp();
#pragma unroll 16
      for (int q = 0; q < 32; ++q)
        if (r0 + lane < nr && c0 + q < nc) G[(long)(r0 + lane) + (long)(c0 + q) * ldg] = tile[lane * 33 + q];
    }
    __syncwarp();
  }
}

template <int NT>
__global__ void __launch_bounds__(NT, LuB<NT>::MINB) lu_batched_f64_kernel(BatchArgs<double> a, double* ws,
                                                                           size_t ws_stride) {
  using S = LuB<NT>;
  constexpr int NW = S::NW, LDU = S::LDU;
  extern __shared__ __align__(16) double lub_sm[];
  double* big = lub_sm;
  double* sL = big;                        // L(r, k) of the panel at sL[r * LSL + k]
  double* sU = big + NT * LSL;             // U(k, c) of a chunk at sU[k * LDU + c]
  double* srow = big + S::BIG;             // [2][LW] pivot row
  double* rowj = srow + 2 * LW;            // [2][LW] row j
  double* sx = rowj + 2 * LW;              // [LMAXRHS][LW]
  RHdr* hdr = reinterpret_cast<RHdr*>(sx + LMAXRHS * LW);  // [2][NW]
  __shared__ int s_next, s_r[LW], s_nlist;
  __shared__ int2 s_list[2 * LW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* W = ws + (size_t)blockIdx.x * ws_stride;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_next = atomicAdd(a.counter, 1);
    __syncthreads();
    if (s_next >= a.count) break;
    const int mi = a.order[s_next];
    const int n = a.n[mi], nrhs = a.B ? a.nrhs : 0;
    const long ld = a.ld[mi];
    const int n32 = lub_n32(n), ldw = n32 + LMAXRHS;
    const int ncol = n32 + (nrhs > 0 ? LMAXRHS : 0);  // columns carried: matrix, right-hand sides
    // [A | B] row-major; the columns between n and n32 and the unused
    // right-hand sides are zero
    lub_transpose<NT, true>(W, ldw, a.A[mi], ld, n, n, big);
    if (n32 > n || nrhs > 0) {
      const int pad = ncol - n;
      for (int e = tid; e < n * pad; e += NT) {
        const int r = e / pad, c = n + e % pad, q = c - n32;
        W[(long)r * ldw + c] = (q >= 0 && q < nrhs) ? a.B[mi][(long)r + (long)q * a.ldb[mi]] : 0.0;
      }
    }
    __syncthreads();
    int first_null = -1;
    for (int j0 = 0; j0 < n; j0 += LW) {
      const int w = min(LW, n - j0), rows = n - j0;
      __syncthreads();  // the previous panel's update is complete
      double rv[1][LW];
      {
        const double* p = W + (long)(j0 + tid) * ldw + j0;
#pragma unroll
        for (int q = 0; q < LW; q += 2) {
          const double2 v = tid < rows ? *reinterpret_cast<const double2*>(p + q) : make_double2(0.0, 0.0);
          rv[0][q] = v.x;
          rv[0][q + 1] = v.y;
        }
      }
      // ---- panel: columns in registers
      double bv = -1.0;
      int bi = INT_MAX, bk = 0;
      if (tid < rows) {
        const double v = fabs(rv[0][0]);
        if (v > bv) { bv = v; bi = tid; }
      }
#pragma unroll 1
      for (int j = 0; j < w; ++j) {
        const int par = j & 1;
        {
          unsigned long long wk = rleaf_key(bv, bi);
          int wi = bi;
          rleaf_argmax_warp(wk, wi);
          if (wi == INT_MAX ? lane == 0 : wi == bi) {
            RHdr h;
            h.key = wk;
            h.row = wi;
            h.pad = 0;
            hdr[par * NW + warp] = h;
          }
          if (tid == j) rleaf_store_row<LW, 1>(rv, 0, rowj + par * LW);
        }
        __syncthreads();
        int r;
        {
          const RHdr* hs = hdr + par * NW + (lane < NW ? lane : 0);
          unsigned long long ck = lane < NW ? hs->key : 0ull;
          r = lane < NW ? hs->row : INT_MAX;
          rleaf_argmax_warp(ck, r);
          if (r != INT_MAX && r == bi) rleaf_store_row<LW, 1>(rv, 0, srow + par * LW);
        }
        __syncthreads();
        const double* u = srow + par * LW;
        const double* oldj = rowj + par * LW;
        if (r == INT_MAX) {  // no orderable entry (NaN): keep row j
          r = j;
          u = oldj;
        }
        const double piv = u[j];
        if (tid == 0) {
          s_r[j] = r;
          a.piv[mi][j0 + j] = r - j;
        }
        bv = -1.0;
        bi = INT_MAX;
        if (piv == 0.0) {
          if (first_null < 0) first_null = j0 + j;
          if (j + 1 < LW && tid < rows && tid > j) {
            const double t = fabs(rleaf_pick_col<LW>(rv[0], j + 1));
            if (t > bv) { bv = t; bi = tid; }
          }
          continue;
        }
        rleaf_column_at<LW, 1>(j, rv, tid, 0, rows, r, u, oldj, 1.0 / piv, bv, bi, bk);
      }
#pragma unroll
      for (int q = 0; q < LW; q += 2)
        *reinterpret_cast<double2*>(sL + tid * LSL + q) = make_double2(rv[0][q], rv[0][q + 1]);
      __syncthreads();
      // the panel's rows (multipliers and U) back to the copy, whole rows at a
      // time
      for (int e = tid; e < rows * (LW / 2); e += NT) {
        const int r = e / (LW / 2), q = 2 * (e % (LW / 2));
        *reinterpret_cast<double2*>(W + (long)(j0 + r) * ldw + j0 + q) = *reinterpret_cast<const double2*>(sL + r * LSL + q);
      }
      // ---- the interchanges on the other columns.  Warp 0 composes the w swaps
      // over 2 LW slots: the panel's first rows (slot = row) and the far rows
      // (slot LW + first swap with it); lane l holds the labels of slots l and
      // LW + l, and the slots whose row changes form the list (row, source).
      if (warp == 0) {
        const int t = lane < w ? s_r[lane] : lane;
        const unsigned same = __match_any_sync(0xffffffffu, t);
        const int first = __ffs(same) - 1;
        const int tgt = t < LW ? t : LW + first;         // slot of row t (rows w.. of a short panel: themselves)
        const int row1 = t >= LW && first == lane ? t : -1;  // row of slot LW + lane
        int d0 = lane, d1 = LW + lane;
        for (int i = 0; i < w; ++i) {
          const int b = __shfl_sync(0xffffffffu, tgt, i);
          const int x = __shfl_sync(0xffffffffu, d0, i);
          const int y0 = __shfl_sync(0xffffffffu, d0, b & 31), y1 = __shfl_sync(0xffffffffu, d1, b & 31);
          const int y = b < LW ? y0 : y1;
          if (lane == i) d0 = y;
          if (lane == (b & 31)) { if (b < LW) d0 = x; else d1 = x; }
        }
        // labels are slots: the row that a slot's content comes from
        auto row_of = [&](int slot) {
          const int far = __shfl_sync(0xffffffffu, row1, slot & 31);
          return slot < LW ? slot : far;
        };
        const int src0 = row_of(d0), src1 = row_of(d1);
        const unsigned m0 = __ballot_sync(0xffffffffu, d0 != lane);
        const unsigned m1 = __ballot_sync(0xffffffffu, row1 >= 0 && d1 != LW + lane);
        const unsigned below = (1u << lane) - 1u;
        if (d0 != lane) s_list[__popc(m0 & below)] = make_int2(lane, src0);
        if (row1 >= 0 && d1 != LW + lane) s_list[__popc(m0) + __popc(m1 & below)] = make_int2(row1, src1);
        if (lane == 0) s_nlist = __popc(m0) + __popc(m1);
      }
      __syncthreads();
      const int m = s_nlist, tot2 = (ncol - LW) / 2;  // changed rows; other columns, in pairs
      if (m > 0) {
        // whole rows through the (free) U12 buffer, one warp per row
        const int cap2 = LW * LDU / 2 / m;  // column pairs per pass
        for (int c2 = 0; c2 < tot2; c2 += cap2) {
          const int k2 = min(cap2, tot2 - c2);
          for (int l = warp; l < m; l += NW) {
            const double* p = W + (long)(j0 + s_list[l].y) * ldw;
#pragma unroll 4
            for (int k = lane; k < k2; k += 32) {
              const int c = 2 * (c2 + k);
              reinterpret_cast<double2*>(sU)[l * k2 + k] = *reinterpret_cast<const double2*>(p + (c < j0 ? c : c + LW));
            }
          }
          __syncthreads();
          for (int l = warp; l < m; l += NW) {
            double* p = W + (long)(j0 + s_list[l].x) * ldw;
#pragma unroll 4
            for (int k = lane; k < k2; k += 32) {
              const int c = 2 * (c2 + k);
              *reinterpret_cast<double2*>(p + (c < j0 ? c : c + LW)) = reinterpret_cast<double2*>(sU)[l * k2 + k];
            }
          }
          __syncthreads();
        }
      }
      const int ct = ncol - j0 - LW;  // trailing columns (a multiple of 8)
      if (ct <= 0) continue;
      // ---- U12: one thread per column
      if (tid < ct) {
        double* p = W + (long)j0 * ldw + j0 + LW + tid;
        double x[LW];
#pragma unroll
        for (int i = 0; i < LW; ++i) x[i] = i < w ? p[(long)i * ldw] : 0.0;
#pragma unroll
        for (int i = 1; i < LW; ++i) {
          double s0 = x[i], s1 = 0.0;
#pragma unroll
          for (int k = 0; k + 1 < i; k += 2) {
            const double2 l = *reinterpret_cast<const double2*>(sL + i * LSL + k);
            s0 = fma(-l.x, x[k], s0);
            s1 = fma(-l.y, x[k + 1], s1);
          }
          if (i & 1) s0 = fma(-sL[i * LSL + i - 1], x[i - 1], s0);
          x[i] = i < w ? s0 + s1 : 0.0;
        }
#pragma unroll
        for (int i = 0; i < LW; ++i)
          if (i < w) p[(long)i * ldw] = x[i];
        if (tid < S::CW)
#pragma unroll
          for (int i = 0; i < LW; ++i) sU[i * LDU + tid] = x[i];
      }
      __syncthreads();
      // ---- A22 -= L21 U12 (w = LW here: there are rows below)
      const int R2 = rows - LW;
      if (R2 <= 0) continue;
      const int g = lane >> 2, t = lane & 3;
      for (int cb = 0; cb < ct; cb += S::CW) {
        const int cw = min(S::CW, ct - cb);
        if (cb > 0) {
          __syncthreads();
          for (int e = tid; e < LW * (cw / 2); e += NT) {
            const int k = e / (cw / 2), c = 2 * (e % (cw / 2));
            *reinterpret_cast<double2*>(sU + k * LDU + c) =
                *reinterpret_cast<const double2*>(W + (long)(j0 + k) * ldw + j0 + LW + cb + c);
          }
          __syncthreads();
        }
        const int tr = (R2 + 15) / 16, tc = (cw + 31) / 32;
        for (int e = warp; e < tr * tc; e += NW) {
          const int r0 = (e % tr) * 16, c0 = (e / tr) * 32;
          const int nct = min(4, (cw - c0) / 8);
          double* C = W + (long)(j0 + LW + r0 + g) * ldw + j0 + LW + cb + c0 + 2 * t;
          double d[2][4][2];
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              double2 v = make_double2(0.0, 0.0);
              if (c < nct) v = *reinterpret_cast<const double2*>(C + (long)(8 * i) * ldw + 8 * c);
              d[i][c][0] = v.x;
              d[i][c][1] = v.y;
            }
          const double* pa = sL + (LW + r0 + g) * LSL + t;
          const double* pb = sU + t * LDU + c0 + g;
#pragma unroll
          for (int k = 0; k < LW; k += 4) {
            // (LW + r0 + 15 < NT: the tile rows end at a multiple of 16)
            const double a0 = -pa[k], a1 = -pa[k + 8 * LSL];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const double b = pb[k * LDU + 8 * c];
              dmma_884(d[0][c][0], d[0][c][1], a0, b);
              dmma_884(d[1][c][0], d[1][c][1], a1, b);
            }
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (c < nct && r0 + 8 * i + g < R2)
                *reinterpret_cast<double2*>(C + (long)(8 * i) * ldw + 8 * c) = make_double2(d[i][c][0], d[i][c][1]);
        }
      }
    }
    __syncthreads();
    if (tid == 0) a.info[mi] = first_null;
    lub_transpose<NT, false>(W, ldw, a.A[mi], ld, n, n, big);
    // ---- backward substitution: the right-hand sides hold inv(L) P B
    if (nrhs > 0 && first_null < 0) {
      double* sD = big;  // 32 x 33 diagonal block
      for (int b0 = (n - 1) / LW * LW; b0 >= 0; b0 -= LW) {
        const int w = min(LW, n - b0);
        __syncthreads();
        // this thread's row above the block (b0 <= NT): in flight during the
        // block's own solve
        double u[LW];
        {
          const double* p = W + (long)tid * ldw + b0;
#pragma unroll
          for (int s = 0; s < LW; s += 2) {
            const double2 x = tid < b0 ? *reinterpret_cast<const double2*>(p + s) : make_double2(0.0, 0.0);
            u[s] = x.x;
            u[s + 1] = x.y;
          }
        }
        for (int e = tid; e < LW * LW; e += NT) {
          const int r = e / LW, c = e % LW;
          sD[r * 33 + c] = r < w && c < w ? W[(long)(b0 + r) * ldw + b0 + c] : (r == c ? 1.0 : 0.0);
        }
        __syncthreads();
        for (int q = warp; q < nrhs; q += NW) {
          double y = lane < w ? W[(long)(b0 + lane) * ldw + n32 + q] : 0.0;
          const double rinv = 1.0 / sD[lane * 33 + lane];
          for (int s = w - 1; s >= 0; --s) {
            const double x = __shfl_sync(0xffffffffu, y * rinv, s);
            if (lane == s) y = x;
            else if (lane < s) y = fma(-sD[lane * 33 + s], x, y);
          }
          sx[q * LW + lane] = y;
          if (lane < w) a.B[mi][(long)(b0 + lane) + (long)q * a.ldb[mi]] = y;
        }
        __syncthreads();
        if (tid < b0) {
          for (int q = 0; q < nrhs; ++q) {
            double y0 = 0.0, y1 = 0.0;  // summed apart: one rounding at the size of the entry
#pragma unroll
            for (int s = 0; s < LW; s += 2) {  // entries past w meet zeros of the copy
              y0 = fma(u[s], sx[q * LW + s], y0);
              y1 = fma(u[s + 1], sx[q * LW + s + 1], y1);
            }
            W[(long)tid * ldw + n32 + q] -= y0 + y1;
          }
        }
      }
    }
  }
}

template <int NT>
int lub_launch(const BatchArgs<double>& a, double* ws, size_t stride, int grid, cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    FB_CK(cudaFuncSetAttribute(lu_batched_f64_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)LuB<NT>::SMEM));
    attr = true;
  }
  lu_batched_f64_kernel<NT><<<grid, NT, LuB<NT>::SMEM, st>>>(a, ws, stride);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

}  // namespace

// The schedule (a.order) is largest first; its first `big` matrices are the
// ones above order 256, maxn the largest order.  a.counter: two words.
int batched_lu_f64(BatchArgs<double> a, int big, int maxn, cudaStream_t st) {
  Context& cx = ctx();
  const int sms = cx.num_sms;
  int g_big = std::min(sms, big), g_small = std::min(2 * sms, a.count - big);
  const size_t s_big = (lub_ws(maxn) + 1) & ~size_t(1);
  const size_t s_small = (lub_ws(std::min(maxn, 256)) + 1) & ~size_t(1);
  // a CTA's copy is 2.2 MB at order 512, 0.5 GB in all for a full GPU; with
  // less memory to be had, fewer CTAs take the matrices
  double* ws;
  while (!(ws = (double*)ws_get(WS_REPACK, sizeof(double) * (s_big * g_big + s_small * g_small)))) {
    if (g_big <= 1 && g_small <= 1) return FLA_FAILURE;
    g_big = (g_big + 1) / 2;
    g_small = (g_small + 1) / 2;
  }
  const int ps = prof_begin(st);
  if (g_small > 0 && g_big > 0) {
    // beside the large ones: their CTAs take the SMs the others leave
    FB_CK(cudaEventRecord(cx.ev[0], st));
    FB_CK(cudaStreamWaitEvent(cx.side, cx.ev[0], 0));
  }
  if (g_big > 0) {
    BatchArgs<double> b = a;
    b.count = big;
    if (lub_launch<512>(b, ws, s_big, g_big, st) != FLA_SUCCESS) return FLA_FAILURE;
  }
  if (g_small > 0) {
    BatchArgs<double> b = a;
    b.count = a.count - big;
    b.order = a.order + big;
    b.counter = a.counter + 1;
    cudaStream_t s2 = g_big > 0 ? cx.side : st;
    if (lub_launch<256>(b, ws + s_big * g_big, s_small, g_small, s2) != FLA_SUCCESS) return FLA_FAILURE;
    if (g_big > 0) {
      FB_CK(cudaEventRecord(cx.ev[1], s2));
      FB_CK(cudaStreamWaitEvent(st, cx.ev[1], 0));
    }
  }
  prof_end(ps, st, PROF_OTHER, 0.0);
  return FLA_SUCCESS;
}

}  // namespace fb
