// Device pieces of the register-resident LU panels (lu_panel.cu, one cluster
// per leaf; batched_lu.cu, one CTA per matrix): candidates, and the column
// step on rows held in registers.
#pragma once
#include <climits>

#include "dev_util.cuh"

namespace fb {

namespace {

constexpr int RLEAF_THREADS = 512;

// A warp's candidate: ordering key and row.
struct RHdr {
  unsigned long long key;
  int row;
  int pad;
};

// Non-negative magnitudes order like their bit patterns, so the key orders
// candidates by magnitude; no candidate orders below every magnitude (and
// NaN never becomes a candidate: `t > best` is false for it).
__device__ __forceinline__ unsigned long long rleaf_key(double bv, int bi) {
  return bi == INT_MAX ? 0ull : (unsigned long long)__double_as_longlong(bv) + 1ull;
}

// Warp argmax of (key, row): the largest key, the smallest row among equal
// keys; every lane receives the result.  Rows are distinct, INT_MAX marks
// no candidate (key 0).
__device__ __forceinline__ void rleaf_argmax_warp(unsigned long long& key, int& row) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  const bool top = hi == mhi && lo == mlo;
  row = (int)__reduce_min_sync(0xffffffffu, top ? (unsigned)row : 0xffffffffu);
  key = ((unsigned long long)mhi << 32) | mlo;
}

template <int W, int RPT>
__device__ __forceinline__ double rleaf_pick(const double (&rv)[RPT][W], int k, int q) {
  double v = rv[0][q];
#pragma unroll
  for (int kk = 1; kk < RPT; ++kk)
    if (kk == k) v = rv[kk][q];
  return v;
}

// Row slot k of the calling thread into shared memory (16-byte aligned).
template <int W, int RPT>
__device__ __forceinline__ void rleaf_store_row(const double (&rv)[RPT][W], int k, double* dst) {
#pragma unroll
  for (int q = 0; q < W; q += 2)
    *reinterpret_cast<double2*>(dst + q) = make_double2(rleaf_pick<W, RPT>(rv, k, q), rleaf_pick<W, RPT>(rv, k, q + 1));
}

// Entry j (run-time) of a register row: a select chain over compile-time
// indices, so the row stays in registers.
template <int W>
__device__ __forceinline__ double rleaf_pick_col(const double (&row)[W], int j) {
  double v = row[0];
#pragma unroll
  for (int q = 1; q < W; ++q)
    if (q == j) v = row[q];
  return v;
}

// Rows j and r of the leaf exchanged: the owner of row j takes the pivot row
// u, the owner of row r the old row j.
template <int W, int RPT>
__device__ __forceinline__ void rleaf_exchange(int j, double (&rv)[RPT][W], int tid, int r0, int rows, int r,
                                               const double* u, const double* oldj) {
  if (r == j) return;
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int i = tid + k * RLEAF_THREADS, gi = r0 + i;
    if (i < rows && (gi == j || gi == r)) {
      const double* src = gi == j ? u : oldj;
#pragma unroll
      for (int q = 0; q < W; q += 2) {
        const double2 v = *reinterpret_cast<const double2*>(src + q);
        rv[k][q] = v.x;
        rv[k][q + 1] = v.y;
      }
    }
  }
}

// Column J of the leaf for the calling thread's rows, J a compile-time
// constant so every register of a row is addressed directly: scale column J
// below the pivot (reciprocal multiply, as bl1_dinvscalv), rank-1 update, and
// the candidate for column J + 1.  A column's body runs once per leaf and
// comes from beyond the SM's instruction caches, so it holds nothing that
// could stand outside it (with the exchange inside, 3000 x 32 took 53.4 us,
// now 51.8; bodies shared by two columns, the column selected at run time,
// 80).
template <int W, int RPT, int J>
__device__ __forceinline__ void rleaf_column(double (&rv)[RPT][W], int tid, int r0, int rows, const double* u,
                                             double rinv, double& bv, int& bi, int& bk) {
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int i = tid + k * RLEAF_THREADS, gi = r0 + i;
    if (i >= rows || gi <= J) continue;
    const double l = rv[k][J] * rinv;
    rv[k][J] = l;
#pragma unroll
    for (int q = (J + 1) & ~1; q < W; q += 2) {
      const double2 v = *reinterpret_cast<const double2*>(u + q);
      if (q > J) rv[k][q] = fma(-l, v.x, rv[k][q]);
      rv[k][q + 1] = fma(-l, v.y, rv[k][q + 1]);
    }
    if constexpr (J + 1 < W) {
      const double t = fabs(rv[k][J + 1]);
      if (t > bv) { bv = t; bi = gi; bk = k; }
    }
  }
}

// The exchange, then run-time column j to its compile-time body through one
// jump table.
template <int W, int RPT>
__device__ __forceinline__ void rleaf_column_at(int j, double (&rv)[RPT][W], int tid, int r0, int rows, int r,
                                                const double* u, const double* oldj, double rinv, double& bv,
                                                int& bi, int& bk) {
  static_assert(W <= 32 && W % 2 == 0, "leaf width");
  rleaf_exchange<W, RPT>(j, rv, tid, r0, rows, r, u, oldj);
  switch (j) {
#define FB_RLEAF_CASE(J)                                                              \
  case J:                                                                             \
    if constexpr (J < W) rleaf_column<W, RPT, J>(rv, tid, r0, rows, u, rinv, bv, bi, bk); \
    break;
    FB_RLEAF_CASE(0) FB_RLEAF_CASE(1) FB_RLEAF_CASE(2) FB_RLEAF_CASE(3) FB_RLEAF_CASE(4) FB_RLEAF_CASE(5)
    FB_RLEAF_CASE(6) FB_RLEAF_CASE(7) FB_RLEAF_CASE(8) FB_RLEAF_CASE(9) FB_RLEAF_CASE(10) FB_RLEAF_CASE(11)
    FB_RLEAF_CASE(12) FB_RLEAF_CASE(13) FB_RLEAF_CASE(14) FB_RLEAF_CASE(15) FB_RLEAF_CASE(16)
    FB_RLEAF_CASE(17) FB_RLEAF_CASE(18) FB_RLEAF_CASE(19) FB_RLEAF_CASE(20) FB_RLEAF_CASE(21)
    FB_RLEAF_CASE(22) FB_RLEAF_CASE(23) FB_RLEAF_CASE(24) FB_RLEAF_CASE(25) FB_RLEAF_CASE(26)
    FB_RLEAF_CASE(27) FB_RLEAF_CASE(28) FB_RLEAF_CASE(29) FB_RLEAF_CASE(30) FB_RLEAF_CASE(31)
#undef FB_RLEAF_CASE
    default:
      break;
  }
}

}  // namespace

}  // namespace fb
