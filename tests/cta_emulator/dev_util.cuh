// Host stand-in for the library's dev_util.cuh: the threads of one CTA as
// fibers on one host thread, so that a kernel body runs under chosen
// schedules.  A thread runs until a barrier, a warp operation or its end;
// the next one is the first runnable thread of `order`.  A body that is free
// of races on shared memory gives the same bits under every order.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <ucontext.h>
#include <vector>

#define __device__
#define __forceinline__ inline

using std::fma;
using std::max;
using std::min;

struct double2 {
  double x, y;
};
inline double rsqrt(double x) { return (double)(1.0L / sqrtl((long double)x)); }

namespace emu {

struct Idx {
  int x;
};
enum State { RUN, BARRIER, WARP, DONE };
struct Thread {
  ucontext_t ctx;
  std::vector<char> stack;
  State state = RUN;
  int bar = 0;           // barrier waited for
  int syncs = 0;         // __syncthreads() passed
  unsigned ops = 0;      // warp operations begun
  double a[2], b[2];     // operands of the last two warp operations
};
inline std::vector<Thread> th;
inline ucontext_t main_ctx;
inline int cur = 0, waiting[16], expected[16];
inline std::function<void()> body;

inline void yield() { swapcontext(&th[cur].ctx, &main_ctx); }
inline void release(State s, int lo, int hi, int bar) {
  for (int i = lo; i < hi; ++i)
    if (th[i].state == s && (s == WARP || th[i].bar == bar)) th[i].state = RUN;
}
inline void check(int bar) {
  int n = expected[bar];
  if (bar == 0) {
    n = 0;
    for (auto& t : th) n += t.state != DONE;
  }
  if (waiting[bar] > 0 && waiting[bar] >= n) {
    waiting[bar] = 0;
    release(BARRIER, 0, (int)th.size(), bar);
  }
}
inline void arrive(int bar, int n, bool wait = true) {
  Thread& t = th[cur];
  if (wait) t.state = BARRIER;
  t.bar = bar;
  expected[bar] = n;
  if (bar == 0) ++t.syncs;
  ++waiting[bar];
  check(bar);
  if (t.state != RUN) yield();
}
// all lanes of the warp have begun this operation; returns its buffer
inline unsigned warp_op(double a, double b) {
  Thread& t = th[cur];
  const unsigned s = t.ops++ & 1;
  t.a[s] = a;
  t.b[s] = b;
  t.state = WARP;
  const int lo = cur & ~31;
  bool all = true;
  for (int i = lo; i < lo + 32; ++i) all = all && th[i].state == WARP && th[i].ops == t.ops;
  if (all) release(WARP, lo, lo + 32, 0);
  else yield();
  return s;
}
inline void entry() {
  body();
  th[cur].state = DONE;
  check(0);
  yield();
}
// Runs f in n threads under the given order; false on a deadlock or when the
// threads did not all pass the same number of CTA barriers.
inline bool run(int n, const std::vector<int>& order, std::function<void()> f) {
  th.clear();
  th.resize(n);
  body = std::move(f);
  for (int b = 0; b < 16; ++b) waiting[b] = expected[b] = 0;
  for (auto& t : th) {
    t.stack.resize(1 << 16);
    getcontext(&t.ctx);
    t.ctx.uc_stack.ss_sp = t.stack.data();
    t.ctx.uc_stack.ss_size = t.stack.size();
    t.ctx.uc_link = nullptr;
    makecontext(&t.ctx, entry, 0);
  }
  for (;;) {
    int next = -1;
    for (int i : order)
      if (th[i].state == RUN) {
        next = i;
        break;
      }
    if (next < 0) break;
    cur = next;
    swapcontext(&main_ctx, &th[next].ctx);
  }
  bool ok = true;
  for (auto& t : th) ok = ok && t.state == DONE && t.syncs == th[0].syncs;
  return ok;
}

}  // namespace emu

#define threadIdx (emu::Idx{emu::cur})
inline void __syncthreads() { emu::arrive(0, 0); }

namespace fb {
inline void bar_sync(int id, int threads) { emu::arrive(id, threads); }
inline void bar_arrive(int id, int threads) { emu::arrive(id, threads, false); }
// D(g, 2t..2t+1) += sum_k A(g, k) B(k, 2t..), lane = 4 g + t holding A(g, t), B(t, g)
inline void dmma_884(double& d0, double& d1, double a, double b) {
  const int lane = emu::cur & 31, lo = emu::cur - lane, g = lane >> 2, t = lane & 3;
  const unsigned s = emu::warp_op(a, b);
  for (int k = 0; k < 4; ++k) {
    const double av = emu::th[lo + 4 * g + k].a[s];
    d0 = fma(av, emu::th[lo + 4 * (2 * t) + k].b[s], d0);
    d1 = fma(av, emu::th[lo + 4 * (2 * t + 1) + k].b[s], d1);
  }
}
}  // namespace fb
