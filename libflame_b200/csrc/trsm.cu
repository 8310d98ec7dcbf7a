// Left triangular solves X := inv(op(T)) X on the GPU: with one diagonal block
// (b <= 128, trsm_block), of a whole triangle in one launch (trsm_sweep), and
// the inverses of triangles and of their diagonal blocks.
//
// Replaces the dtrsm_ calls of the reference's blocked algorithms
// (FLA_Trsm_external, src/base/flamec/wrappers/blas/3/external/
// FLA_Trsm_external.c:72).  Substitution order follows dtrsm: forward when
// op(T) is lower, backward when upper; non-unit diagonals are applied as a
// multiplication by the reciprocal of the pivot (as dtrsm's R,L,T,N case,
// src/flablas/f2c/dtrsm.c).
//
// trsm_block: one CTA owns 64 columns of X, kept in shared memory with the
// triangle, and sweeps the b steps: scale the current unknown (one thread per
// right-hand side), then update the remaining unknowns (all threads).  The step
// loop is not unrolled, so the kernel stays small in the instruction cache.
#include <algorithm>

#include "common.h"
#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int TB = 128;             // max triangle order
constexpr int NV = 64;              // right-hand sides per CTA
constexpr int THREADS = 256;
constexpr int LDT = TB + 1;         // SMEM stride of the triangle
constexpr int LDX = TB + 1;         // SMEM stride of one right-hand side
constexpr size_t SMEM = (size_t)(TB * LDT + NV * LDX + NV + TB) * sizeof(double);

// coef(r, j): entry of op(T) at (r, j), from the stored triangle S
template <bool TRANS>
__device__ __forceinline__ double coef(const double* S, int r, int j) {
  return TRANS ? S[j + r * LDT] : S[r + j * LDT];
}

template <bool LOWER, bool TRANS, bool UNIT>
__global__ void __launch_bounds__(THREADS) trsm_tile_kernel(const double* __restrict__ T, long ldt,
                                                            double* __restrict__ X, long ldx, int b,
                                                            int nvec) {
  extern __shared__ double sm[];
  double* ST = sm;                    // b x b triangle (stored part only)
  double* SX = ST + TB * LDT;         // NV right-hand sides, SX[r + v*LDX]
  double* sx = SX + NV * LDX;         // scaled current unknown per rhs
  double* sd = sx + NV;               // reciprocal diagonal
  constexpr bool FWD = (LOWER != TRANS);
  const int tid = threadIdx.x;
  const int v0 = blockIdx.x * NV;
  const int nv = min(NV, nvec - v0);
  load_block_f64<THREADS, true>(T, ldt, b, ST, LDT, [](int r, int c) { return LOWER ? (r >= c) : (r <= c); });
  for (int v = tid >> 5; v < nv; v += THREADS / 32)
    for (int r = tid & 31; r < b; r += 32) SX[r + v * LDX] = X[r + (long)(v0 + v) * ldx];
  __syncthreads();
  if (!UNIT)
    for (int j = tid; j < b; j += THREADS) sd[j] = 1.0 / ST[j + j * LDT];
  __syncthreads();
  for (int jj = 0; jj < b; ++jj) {
    const int j = FWD ? jj : (b - 1 - jj);
    if (tid < nv) {
      double x = SX[j + tid * LDX];
      if (!UNIT) {
        x *= sd[j];
        SX[j + tid * LDX] = x;
      }
      sx[tid] = x;
    }
    __syncthreads();
    // remaining unknowns: FWD r in (j, b), BWD r in [0, j)
    const int r_lo = FWD ? j + 1 : 0;
    const int cnt = (FWD ? (b - j - 1) : j) * nv;
    if (nv == NV) {
      for (int e = tid; e < cnt; e += THREADS) {
        const int r = r_lo + (e >> 6), v = e & (NV - 1);
        SX[r + v * LDX] -= coef<TRANS>(ST, r, j) * sx[v];
      }
    } else {
      for (int e = tid; e < cnt; e += THREADS) {
        const int r = r_lo + e / nv, v = e % nv;
        SX[r + v * LDX] -= coef<TRANS>(ST, r, j) * sx[v];
      }
    }
    __syncthreads();
  }
  for (int v = tid >> 5; v < nv; v += THREADS / 32)
    for (int r = tid & 31; r < b; r += 32) X[r + (long)(v0 + v) * ldx] = SX[r + v * LDX];
}

// X := inv(T) for a b x b triangular T (b <= 128), one warp per column of X.
// Column c of inv(T) solves T x = e_c: the warp keeps the running right-hand
// side in registers (lane l holds rows l, l+32, l+64, l+96), and at each step
// the owner of the current unknown broadcasts it (multiplied by the
// reciprocal of the pivot unless UNIT) and every lane updates its rows with
// one column of T from shared memory.  No block barriers inside the sweep,
// so the b steps cost only warp-level latency.
constexpr int INV_WARPS = 16;
constexpr size_t inv_smem(int bs) { return (size_t)(bs * LDT + TB) * sizeof(double); }
constexpr size_t INV_SMEM = inv_smem(TB);
// Batched over the diagonal blocks of order bs (<= TB) of an n x n
// triangle: blockIdx.y = block index q, T_q = T + q*bs*(1 + ldt), X_q = X +
// q * xstride; with gridDim.y = 1 and n = b, the single b x b block.
template <bool LOWER, bool UNIT>
__global__ void __launch_bounds__(INV_WARPS * 32) tri_inv_kernel(const double* __restrict__ T, long ldt,
                                                                 double* __restrict__ X, long ldx, int n,
                                                                 long xstride, int bs = TB) {
  extern __shared__ double sm[];
  double* ST = sm;             // stored triangle, ST[r + c*LDT]
  double* sd = ST + bs * LDT;  // reciprocal diagonal
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q = blockIdx.y;
  const int b = min(bs, n - q * bs);
  T += (long)q * bs * (1 + ldt);
  X += (long)q * xstride;
  load_block_f64<INV_WARPS * 32, true>(T, ldt, b, ST, LDT, [](int r, int c) { return LOWER ? (r >= c) : (r <= c); });
  __syncthreads();
  if (!UNIT)
    for (int j = tid; j < b; j += INV_WARPS * 32) sd[j] = 1.0 / ST[j + j * LDT];
  __syncthreads();
  const int c = blockIdx.x * INV_WARPS + warp;
  if (c >= b) return;
  double r[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) r[m] = (lane + 32 * m == c) ? 1.0 : 0.0;
  const int j_first = c, j_last = LOWER ? b - 1 : 0;
  const int nsteps = LOWER ? (b - c) : (c + 1);
  for (int s = 0; s < nsteps; ++s) {
    const int j = LOWER ? j_first + s : j_first - s;
    const int slot = j >> 5;
    double v = r[0];
#pragma unroll
    for (int m = 1; m < 4; ++m)
      if (slot == m) v = r[m];
    double xj = __shfl_sync(0xffffffffu, v, j & 31);
    if (!UNIT) xj *= sd[j];
    // branch-free: rows outside the triangle multiply a zero of ST
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int i = lane + 32 * m;
      const double t = r[m] - ST[i + j * LDT] * xj;
      r[m] = (i == j) ? xj : ((LOWER ? (i > j) : (i < j)) ? t : r[m]);
    }
  }
  (void)j_last;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int i = lane + 32 * m;
    if (i < b) X[i + (long)c * ldx] = (LOWER ? i >= c : i <= c) ? r[m] : 0.0;
  }
}


// ---------------------------------------------------------------------------
// Whole blocked triangular solve B := inv(op(T)) B in one cooperative launch
// (FP64): 64-row blocks, groups of 16 right-hand sides.
//
//   X_q := op(Inv_q) (Y_q - sum_{j solved before q} op(T)(q, j) X_j)
//
// A task is one block row for one group of columns; tasks are numbered in
// solve order (all groups of a row, then the next row) and CTA c takes tasks
// c, c + gridDim.x, ..., so the lowest unfinished task never waits for one
// that has not been taken.  The solve is bound by its chain: a block's last
// product needs the block solved just before it.  So everything else is done
// while the chain advances: the tiles of op(T) stream through two half-tile
// buffers (cp.async, 64 x 32 each), the inverse sits in shared memory, and
// solved blocks pass between CTAs through an exchange buffer whose entries
// start as all-ones (a NaN no arithmetic produces): a reader polls the data
// itself, one trip through L2 per step instead of store, fence, flag, poll
// and load.  Per step of the chain: that trip and two 64 x 64 x 16 DMMA
// products.  n = 8192, 32 columns: 3.0 us per block (FP64 factors), 2.7 us
// (FP32).
// ---------------------------------------------------------------------------
constexpr int SB = 64;                  // block rows
constexpr int SC = 16;                  // right-hand sides per task
constexpr int SH = SB / 2;              // k-width of a half tile
constexpr int SLD = SB + 4;             // X, Z: = 4 mod 16, conflict-free fragments
// Tiles of op(T) and the inverse in the factor's type TF, in either storage:
// row index contiguous (ld RI) or k contiguous (ld KH for a half tile, KF for
// the inverse).  A fragment load touches rows g = 0..7 and k = t = 0..3 (half
// of them at a time for doubles): conflict-free with RI = 4 mod 16 doubles or 8
// mod 32 floats, KH, KF = 4 mod 16 doubles or 4 mod 32 floats.
template <typename TF>
struct SweepTile {
  static constexpr int RI = sizeof(TF) == 8 ? SB + 4 : SB + 8;
  static constexpr int KH = SH + 4, KF = SB + 4;
  static constexpr int HALF = SB * KH > SH * RI ? SB * KH : SH * RI;
  static constexpr int FULL = SB * (RI > KF ? RI : KF);
  static constexpr size_t SMEM = sizeof(TF) * (2 * HALF + FULL) + sizeof(double) * 2 * SC * SLD;
};

template <typename TF, typename TV>
struct SweepArgs {
  const TF* T;     // n x n triangle, ld ldt
  long ldt;
  const TF* Inv;   // inverse of block q at Inv + (q / per) * istride + (q % per) * SB * (1 + ldi), ld ldi
  long ldi, istride;
  int per;
  const TV* Y;     // right-hand sides (ld ldb); may be X
  TV* X;           // solutions (ld ldb)
  long ldb;
  double* XB;      // exchange buffer, nblk * SB x nr, all ones
  int n, nr, nblk;
  int* err;
  int first;       // first task: 0 (the check of the waits leaves the first block unsolved)
};

// TRANS: op(T)(r, c) = T(c, r), op(Inv) alike.  BWD: blocks solved last to
// first.  Products and sums in FP64 for either type of factor.
template <bool TRANS, bool BWD, typename TF, typename TV>
__global__ void __launch_bounds__(256, 2) trsm_sweep_kernel(SweepArgs<TF, TV> a) {
  using ST = SweepTile<TF>;
  constexpr int V = 16 / sizeof(TF);    // elements per copy
  extern __shared__ __align__(16) unsigned char sw_sm[];
  double* sX = reinterpret_cast<double*>(sw_sm);  // X_j: sX[k + c * SLD]
  double* sZ = sX + SC * SLD;                     // Y_q - sum
  TF* sT = reinterpret_cast<TF*>(sZ + SC * SLD);  // two half tiles
  TF* sI = sT + 2 * ST::HALF;                     // op(Inv_q)
  __shared__ int s_dead;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int i0 = warp * 8 + g;          // this lane's row of the block
  const int n = a.n, nr = a.nr, nblk = a.nblk;
  const int ngrp = (nr + SC - 1) / SC;
  const long ldx = (long)nblk * SB;     // exchange buffer: padded rows x columns
  if (tid == 0) s_dead = 0;
  __syncthreads();
  // an mr x mk block stored row index contiguous (TRANS: k contiguous) at
  // src, ld lds, into dst; rows past vr and columns past vk read as zero
  auto load_tile = [&](const TF* src, long lds, int mk, int vr, int vk, TF* dst, int ldk) {
    if (TRANS) {
      for (int e = tid; e < SB * (mk / V); e += 256) {
        const int k = (e % (mk / V)) * V, i = e / (mk / V);
        const int left = i < vr ? min(V, max(0, vk - k)) : 0;
        cp_async16(dst + k + i * ldk, left > 0 ? src + k + (long)i * lds : src, left * (int)sizeof(TF));
      }
    } else {
      for (int e = tid; e < (SB / V) * mk; e += 256) {
        const int i = (e % (SB / V)) * V, k = e / (SB / V);
        const int left = k < vk ? min(V, max(0, vr - i)) : 0;
        cp_async16(dst + i + k * ST::RI, left > 0 ? src + i + (long)k * lds : src, left * (int)sizeof(TF));
      }
    }
  };
  // half tile h of op(T)(block bi, block bj)
  auto load_half = [&](int bi, int bj, int h, TF* buf) {
    const int r0 = bi * SB, c0 = bj * SB + h * SH;
    const TF* src = a.T + (TRANS ? c0 + (long)r0 * a.ldt : r0 + (long)c0 * a.ldt);
    if (c0 < n) load_tile(src, a.ldt, SH, n - r0, n - c0, buf, ST::KH);
    else load_tile(a.T, a.ldt, SH, 0, 0, buf, ST::KH);
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  // the 64 x 16 block X_bj of this group from the exchange buffer, as soon as
  // every entry has been published (bounded wait)
  auto poll_x = [&](int bj, int col0, int nc) {
    const int c = tid >> 4, k0 = (tid & 15) * 4;  // column, four consecutive rows
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (c < nc) {
      const double* p = a.XB + (long)bj * SB + k0 + (long)(col0 + c) * ldx;
      unsigned long long start = 0;
      int spins = 0;
      for (;;) {
        bool all = true;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v[u]) : "l"(p + u) : "memory");
          all = all && __double_as_longlong(v[u]) != -1ll;
        }
        if (all) break;
        if (++spins >= 64) {
          spins = 0;
          const unsigned long long now = globaltimer_ns();
          if (start == 0) start = now;
          if (*((volatile int*)&s_dead) || now - start > kWaitLimitNs) {
            atomicExch(a.err, 52);
            *((volatile int*)&s_dead) = 1;
            break;
          }
        }
      }
    }
    double* d = sX + k0 + c * SLD;
    *reinterpret_cast<double2*>(d) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(d + 2) = make_double2(v[2], v[3]);
  };
  for (int task = blockIdx.x + a.first; task < nblk * ngrp; task += gridDim.x) {
    const int q = task / ngrp, col0 = (task % ngrp) * SC, nc = min(SC, nr - col0);
    const int bi = BWD ? nblk - 1 - q : q, r0 = bi * SB;
    auto blk = [&](int j) { return BWD ? nblk - 1 - j : j; };
    __syncthreads();  // the buffers of the previous task are free
    load_tile(a.Inv + (bi / a.per) * a.istride + (long)(bi % a.per) * SB * (1 + a.ldi), a.ldi, SB, n - r0, n - r0, sI,
              ST::KF);
    commit();
    if (q > 0) load_half(bi, blk(0), 0, sT);
    commit();
    double y[2][2];  // the right-hand sides: read before any solution of this block is stored
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * h + 2 * t + e;
        y[h][e] = (r0 + i0 < n && c < nc) ? (double)a.Y[(long)(r0 + i0) + (long)(col0 + c) * a.ldb] : 0.0;
      }
    // acc[n-tile][parity of the k-step]: four chains of DMMAs
    double acc[2][2][2] = {};
    for (int u = 0; u < 2 * q; ++u) {
      if (u + 1 < 2 * q) load_half(bi, blk((u + 1) >> 1), (u + 1) & 1, sT + ((u + 1) & 1) * ST::HALF);
      commit();
      if ((u & 1) == 0) poll_x(blk(u >> 1), col0, nc);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      const TF* buf = sT + (u & 1) * ST::HALF;
      const TF* pa = TRANS ? buf + t + i0 * ST::KH : buf + i0 + t * ST::RI;
      const double* pb = sX + (u & 1) * SH + t + g * SLD;
#pragma unroll
      for (int k = 0; k < SH; k += 4) {
        const double x = (double)(TRANS ? pa[k] : pa[k * ST::RI]);
        const double b0 = pb[k], b1 = pb[k + 8 * SLD];
        dmma_884(acc[0][(k >> 2) & 1][0], acc[0][(k >> 2) & 1][1], x, b0);
        dmma_884(acc[1][(k >> 2) & 1][0], acc[1][(k >> 2) & 1][1], x, b1);
      }
      if (u & 1) {
        // a tile's sum leaves the right-hand side at once: one sum over all
        // tiles doubled the error of the solution (one system of n = 8192:
        // 6.4e-13 against 3.0e-13).  Over sixteen systems with the same factors:
        // 2.95e-13, 3.16e-13 with the blocked updates this kernel replaced
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            y[h][e] -= acc[h][0][e] + acc[h][1][e];
            acc[h][0][e] = acc[h][1][e] = 0.0;
          }
      }
      __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sZ[i0 + (8 * h + 2 * t + e) * SLD] = y[h][e];
      }
    __syncthreads();
    // op(Inv)(i, k): Inv(i, k), or Inv(k, i) when transposed
    const TF* pa = TRANS ? sI + t + i0 * ST::KF : sI + i0 + t * ST::RI;
    const double* pb = sZ + t + g * SLD;
#pragma unroll
    for (int k = 0; k < SB; k += 4) {
      const double x = (double)(TRANS ? pa[k] : pa[k * ST::RI]);
      const double b0 = pb[k], b1 = pb[k + 8 * SLD];
      dmma_884(acc[0][(k >> 2) & 1][0], acc[0][(k >> 2) & 1][1], x, b0);
      dmma_884(acc[1][(k >> 2) & 1][0], acc[1][(k >> 2) & 1][1], x, b1);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * h + 2 * t + e;
        double x = acc[h][0][e] + acc[h][1][e];
        if (__double_as_longlong(x) == -1ll) x = __longlong_as_double(0x7ff8000000000000ll);  // another NaN
        if (c < nc) {
          asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(a.XB + (long)r0 + i0 + (long)(col0 + c) * ldx),
                       "d"(x)
                       : "memory");
          if (r0 + i0 < n) a.X[(long)(r0 + i0) + (long)(col0 + c) * a.ldb] = (TV)x;
        }
      }
  }
}

template <bool L, bool T, bool U>
void set_attr_one() {
  cudaFuncSetAttribute(trsm_tile_kernel<L, T, U>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
}

bool g_attr = false;
void set_attrs() {
  if (g_attr) return;
  set_attr_one<true, false, true>();
  set_attr_one<true, false, false>();
  set_attr_one<true, true, true>();
  set_attr_one<true, true, false>();
  set_attr_one<false, false, true>();
  set_attr_one<false, false, false>();
  set_attr_one<false, true, true>();
  set_attr_one<false, true, false>();
  cudaFuncSetAttribute(tri_inv_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)INV_SMEM);
  cudaFuncSetAttribute(tri_inv_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)INV_SMEM);
  cudaFuncSetAttribute(tri_inv_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)INV_SMEM);
  cudaFuncSetAttribute(tri_inv_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)INV_SMEM);
  g_attr = true;
}

}  // namespace

template <typename TF, typename TV>
int sweep_launch(SweepArgs<TF, TV> a, bool trans, bool bwd, cudaStream_t st) {
  void* const kern = bwd ? (trans ? (void*)trsm_sweep_kernel<true, true, TF, TV> : (void*)trsm_sweep_kernel<false, true, TF, TV>)
                         : (trans ? (void*)trsm_sweep_kernel<true, false, TF, TV> : (void*)trsm_sweep_kernel<false, false, TF, TV>);
  constexpr size_t smem = SweepTile<TF>::SMEM;
  static int resident = 0;
  if (resident == 0) {
    int per = 0;
    for (void* f : {(void*)trsm_sweep_kernel<true, true, TF, TV>, (void*)trsm_sweep_kernel<false, true, TF, TV>,
                    (void*)trsm_sweep_kernel<true, false, TF, TV>, (void*)trsm_sweep_kernel<false, false, TF, TV>}) {
      FB_CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      int p = 0;
      FB_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, f, 256, smem));
      per = per == 0 ? p : std::min(per, p);
    }
    resident = std::max(1, per) * ctx().num_sms;
  }
  a.nblk = (a.n + SB - 1) / SB;
  const long tasks = (long)a.nblk * ((a.nr + SC - 1) / SC);
  const size_t xbytes = sizeof(double) * (size_t)a.nblk * SB * (size_t)a.nr;
  a.XB = (double*)ws_get(WS_SOLVE_W, xbytes);
  if (!a.XB) return FLA_FAILURE;
  FB_CK(cudaMemsetAsync(a.XB, 0xff, xbytes, st));
  a.err = ctx().d_status + ST_SOLVE;
  ctx().solve_pending = true;
  void* args[] = {(void*)&a};
  const int ps = prof_begin(st);
  FB_CK(cudaLaunchCooperativeKernel(kern, dim3((unsigned)std::min<long>(tasks, resident)), dim3(256), args, smem, st));
  prof_end(ps, st, PROF_TRSM, (double)a.n * a.n * a.nr);
  count_launch();
  return FLA_SUCCESS;
}

// B := inv(op(T)) B by trsm_sweep_kernel: T n x n, B n x nr, T 16-byte
// aligned with an even leading dimension.  first_task > 0: only for
// solve_wait_check.
int trsm_sweep(DMat T, DMat B, bool lower, bool trans, bool unit, cudaStream_t st, int first_task) {
  const long n = T.m, nblk = (n + SB - 1) / SB;
  double* Inv = (double*)ws_get(WS_TRINV, sizeof(double) * (size_t)nblk * SB * SB);
  if (!Inv) return FLA_FAILURE;
  if (tri_inverse_blocks_bs(T.p, T.ld, n, SB, lower, unit, Inv, st) != FLA_SUCCESS) return FLA_FAILURE;
  SweepArgs<double, double> a = {};
  a.T = T.p;
  a.ldt = T.ld;
  a.Inv = Inv;
  a.ldi = SB;
  a.istride = SB * SB;
  a.per = 1;
  a.Y = B.p;
  a.X = B.p;
  a.ldb = B.ld;
  a.n = (int)n;
  a.nr = (int)B.n;
  a.first = first_task;
  return sweep_launch(a, trans, lower == trans, st);
}

// X := inv(op(F)) Y for the FP32 factors of the mixed-precision solvers, in
// FP64 inside: F n x n (ld ldf a multiple of 4), Inv the FP32 inverses of its
// 128 x 128 diagonal blocks (128 * 128 apart, ld 128; the diagonal halves of
// a triangle's inverse are the inverses of its diagonal halves), X, Y n x nr
// with leading dimension ldb.
int trsm_sweep_f32(const float* F, long ldf, const float* Inv, const float* Y, float* X, long ldb, long n, long nr,
                   bool trans, bool bwd, cudaStream_t st) {
  SweepArgs<float, float> a = {};
  a.T = F;
  a.ldt = ldf;
  a.Inv = Inv;
  a.ldi = 2 * SB;
  a.istride = 4 * SB * SB;
  a.per = 2;
  a.Y = Y;
  a.X = X;
  a.ldb = ldb;
  a.n = (int)n;
  a.nr = (int)nr;
  return sweep_launch(a, trans, bwd, st);
}

// B := inv(op(T)) B for a b x n block B, T b x b (b <= 128) triangular.
int trsm_block(const double* T, long ldt, double* B, long ldb, int b, long n, bool lower, bool trans,
               bool unit, cudaStream_t st) {
  set_attrs();
  if (n <= 0 || b <= 0) return FLA_SUCCESS;
  const unsigned grid = (unsigned)((n + NV - 1) / NV);
  const int ps = prof_begin(st);
#define FB_TRSM_LAUNCH(L, T_, U) \
  trsm_tile_kernel<L, T_, U><<<grid, THREADS, SMEM, st>>>(T, ldt, B, ldb, b, (int)n)
  if (lower) {
    if (!trans) { if (unit) FB_TRSM_LAUNCH(true, false, true); else FB_TRSM_LAUNCH(true, false, false); }
    else        { if (unit) FB_TRSM_LAUNCH(true, true, true);  else FB_TRSM_LAUNCH(true, true, false); }
  } else {
    if (!trans) { if (unit) FB_TRSM_LAUNCH(false, false, true); else FB_TRSM_LAUNCH(false, false, false); }
    else        { if (unit) FB_TRSM_LAUNCH(false, true, true);  else FB_TRSM_LAUNCH(false, true, false); }
  }
#undef FB_TRSM_LAUNCH
  prof_end(ps, st, PROF_TRSM, (double)b * (double)b * (double)n);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}


__global__ void set_identity_kernel(double* X, long ldx, int n) {
  const long total = (long)n * n;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long r = e % n, c = e / n;
    X[r + c * ldx] = (r == c) ? 1.0 : 0.0;
  }
}

// X := inv(L) for the b x b lower-triangular L (unit diagonal if `unit`),
// X b x b with leading dimension ldx: X := I, then the blocked left solve
// L X = I (128-row diagonal solves and GEMM updates).  Used to turn the
// factorizations' panel triangular solves into DMMA GEMMs.
int tri_inverse_lower(const double* L, long ldl, int b, bool unit, double* X, long ldx, cudaStream_t st) {
  return tri_inverse(L, ldl, b, true, unit, X, ldx, st);
}


// X := inv(T) for a b x b triangular T: one warp per column when b <= 128,
// else X := I and the blocked left solve.
int tri_inverse(const double* T, long ldt, int b, bool lower, bool unit, double* X, long ldx, cudaStream_t st) {
  if (b <= 0) return FLA_SUCCESS;
  if (b <= TB) {
    set_attrs();
    const unsigned grid = (unsigned)((b + INV_WARPS - 1) / INV_WARPS);
    const int ps = prof_begin(st);
    if (lower) {
      if (unit) tri_inv_kernel<true, true><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, ldx, b, 0);
      else tri_inv_kernel<true, false><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, ldx, b, 0);
    } else {
      if (unit) tri_inv_kernel<false, true><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, ldx, b, 0);
      else tri_inv_kernel<false, false><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, ldx, b, 0);
    }
    prof_end(ps, st, PROF_TRSM, (double)b * b * b / 3.0);
    count_launch();
    FB_CK(cudaGetLastError());
    return FLA_SUCCESS;
  }
  const int blocks = (int)std::min<long>(1024, ((long)b * b + 255) / 256);
  set_identity_kernel<<<blocks, 256, 0, st>>>(X, ldx, b);
  count_launch();
  FB_CK(cudaGetLastError());
  DMat Tm, B;
  Tm.p = const_cast<double*>(T);
  Tm.ld = ldt;
  Tm.m = Tm.n = b;
  B.p = X;
  B.ld = ldx;
  B.m = B.n = b;
  return trsm_left_dev(Tm, B, lower, false, unit, st);
}


// Inverses of all 128 x 128 diagonal blocks of the n x n triangle T in one
// launch: block q (order min(128, n - 128 q)) into X + q * 128 * 128, ld 128.
int tri_inverse_blocks(const double* T, long ldt, long n, bool lower, bool unit, double* X, cudaStream_t st) {
  if (n <= 0) return FLA_SUCCESS;
  set_attrs();
  const long nblk = (n + TB - 1) / TB;
  dim3 grid((unsigned)((TB + INV_WARPS - 1) / INV_WARPS), (unsigned)nblk);
  const long xs = (long)TB * TB;
  const int ps = prof_begin(st);
  if (lower) {
    if (unit) tri_inv_kernel<true, true><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, TB, (int)n, xs);
    else tri_inv_kernel<true, false><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, TB, (int)n, xs);
  } else {
    if (unit) tri_inv_kernel<false, true><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, TB, (int)n, xs);
    else tri_inv_kernel<false, false><<<grid, INV_WARPS * 32, INV_SMEM, st>>>(T, ldt, X, TB, (int)n, xs);
  }
  prof_end(ps, st, PROF_TRSM, (double)n * TB * TB / 3.0);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

// Inverses of the bs x bs diagonal blocks (bs <= 128) of the n x n
// triangle T in one launch: block q (order min(bs, n - bs q)) into
// X + q * bs * bs, ld bs.
int tri_inverse_blocks_bs(const double* T, long ldt, long n, int bs, bool lower, bool unit, double* X,
                          cudaStream_t st) {
  if (n <= 0) return FLA_SUCCESS;
  set_attrs();
  const long nblk = (n + bs - 1) / bs;
  dim3 grid((unsigned)((bs + INV_WARPS - 1) / INV_WARPS), (unsigned)nblk);
  const long xs = (long)bs * bs;
  const int ps = prof_begin(st);
  if (lower) {
    if (unit) tri_inv_kernel<true, true><<<grid, INV_WARPS * 32, inv_smem(bs), st>>>(T, ldt, X, bs, (int)n, xs, bs);
    else tri_inv_kernel<true, false><<<grid, INV_WARPS * 32, inv_smem(bs), st>>>(T, ldt, X, bs, (int)n, xs, bs);
  } else {
    if (unit) tri_inv_kernel<false, true><<<grid, INV_WARPS * 32, inv_smem(bs), st>>>(T, ldt, X, bs, (int)n, xs, bs);
    else tri_inv_kernel<false, false><<<grid, INV_WARPS * 32, inv_smem(bs), st>>>(T, ldt, X, bs, (int)n, xs, bs);
  }
  prof_end(ps, st, PROF_TRSM, (double)n * bs * bs / 3.0);
  count_launch();
  FB_CK(cudaGetLastError());
  return FLA_SUCCESS;
}

}  // namespace fb
