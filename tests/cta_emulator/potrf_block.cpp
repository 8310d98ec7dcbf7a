// potrf_block (chol_leaf.cuh) under ascending, descending and shuffled thread
// orders.  One line per block order b and failing column f (-1: none):
//   b f return agree barriers error
// agree: the same factor and return value under every order; barriers: every
// thread passed the same CTA barriers; error: largest |L - L_exact| over the
// columns before f, over max |L|, among all orders.
#include <numeric>
#include <random>

#include "chol_leaf.cuh"

int main() {
  using namespace fb;
  std::mt19937_64 rng(5);
  std::normal_distribution<double> nd;
  const int cases[][2] = {{1, -1}, {7, -1}, {8, -1}, {9, -1}, {32, -1}, {33, -1}, {63, -1}, {72, -1}, {100, -1}, {128, -1},
                          {9, 8}, {40, 0}, {72, 35}, {128, 7}, {128, 8}, {128, 77}, {128, 127}};
  for (auto& cs : cases) {
    const int b = cs[0], f = cs[1], ld = POTRF_LD;
    std::vector<double> G(b * b), S0(POTRF_MAX * ld, std::nan(""));
    for (auto& g : G) g = nd(rng);
    for (int c = 0; c < b; ++c)
      for (int r = c; r < b; ++r) {
        double s = r == c ? 1.0 : 0.0;
        for (int k = 0; k < b; ++k) s += G[r + k * b] * G[c + k * b] / b;
        S0[r + c * ld] = s;
      }
    if (f >= 0) S0[f + f * ld] = -1.0;
    std::vector<long double> L(b * b, 0.0L);
    long double top = 0.0L;
    for (int c = 0; c < (f >= 0 ? f : b); ++c)
      for (int r = c; r < b; ++r) {
        long double s = S0[r + c * ld];
        for (int k = 0; k < c; ++k) s -= L[r + k * b] * L[c + k * b];
        L[r + c * b] = r == c ? sqrtl(s) : s / L[c + c * b];
        top = max(top, fabsl(L[r + c * b]));
      }
    std::vector<double> first;
    int ret0 = -2;
    bool agree = true, bars = true;
    long double err = 0.0L;
    for (int o = 0; o < 6; ++o) {
      std::vector<int> order(POTRF_THREADS);
      std::iota(order.begin(), order.end(), 0);
      if (o == 1) std::reverse(order.begin(), order.end());
      if (o > 1) std::shuffle(order.begin(), order.end(), rng);
      alignas(16) static double S[POTRF_MAX * POTRF_LD];
      std::copy(S0.begin(), S0.end(), S);
      int s_fail[2] = {-1, -1};
      std::vector<int> ret(POTRF_THREADS, -2);
      bars = emu::run(POTRF_THREADS, order, [&] {
        const int r = potrf_block(S, b, s_fail);
        ret[emu::cur] = r;
      }) && bars;
      std::vector<double> out;
      for (int c = 0; c < (f >= 0 ? f : b); ++c)
        for (int r = c; r < b; ++r) {
          out.push_back(S[r + c * ld]);
          const long double e = fabsl(S[r + c * ld] - L[r + c * b]);
          err = e <= err ? err : e;  // NaN counts
        }
      if (o == 0) first = out, ret0 = ret[0];
      agree = agree && out == first;
      for (int r : ret) agree = agree && r == ret0;
    }
    printf("%d %d %d %d %d %.3Le\n", b, f, ret0, (int)agree, (int)bars, top > 0 ? err / top : 0.0L);
  }
  return 0;
}
