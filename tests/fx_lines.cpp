// Host driver of the fixed-point line transforms (csrc/fx.cuh) for
// test_fx_lines.py: the kernel's steps on one complex line, thread by thread.
#include <algorithm>
#include <cmath>
#include <vector>

#include "../lattice-dev_gb300/csrc/fx_host.hpp"

using namespace lat::fx;

// in, out: lines A then B of n points, n = N or padded to N
template <int N>
static void line(int n, const double* in, double dk2, double* out) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1;
  std::vector<Tw> w(N), t1(N), t2(N);
  roots(N, w.data());
  for (int i = 0; i < N; ++i) {
    t1[i] = w[(i / P) * (i % P) % N];
    t2[i] = w[(i / Q) * (i % Q) % N];
  }
  std::vector<Mult> H(N / 2 + 1);
  if (n != N) multiplier(n, N, w.data(), H.data());
  int em[2];
  LineBits lb[2];
  std::vector<i64> v[2];
  for (int l = 0; l < 2; ++l) {  // (scaled below: drop_bits may lower a line's scale)
    const double* x = in + l * n;
    em[l] = 1;
    for (int i = 0; i < n; ++i) em[l] = std::max(em[l], exp_of(double_bits(x[i])));
    const i64 x0 = from_bits(double_bits(x[0]), em[l]);
    u64 ored = 0, sum = 0;
    v[l].resize(N);
    for (int i = 0; i < N; ++i) {
      const i64 d = i < n ? from_bits(double_bits(x[i]), em[l]) - x0 : 0;
      const u64 m = (u64)(d ^ (d >> 63));
      v[l][i] = d;
      ored |= m;
      sum += (m >> 9) + 1;
    }
    lb[l] = line_bits<N>(ored, sum);
  }
  const int drop = drop_bits<N>(lb[0], lb[1]);
  for (int l = 0; l < 2; ++l)
    for (int i = 0; i < N; ++i) v[l][i] = scale_line(v[l][i], lb[l]);
  std::vector<Cx64> sl(Q * S);
  for (int t = 0; t < P; ++t) {
    i64 re[Q], im[Q];
    for (int q = 0; q < Q; ++q) {
      re[q] = v[0][t + P * q];
      im[q] = v[1][t + P * q];
    }
    phase1<N>(re, im, t, sl.data(), t1.data());
  }
  for (int t = 0; t < P; ++t) {
    if (n == N) phase2<N>(t, sl.data(), t2.data(), drop);
    else phase2_tab<N>(t, sl.data(), t2.data(), H.data(), drop);
  }
  for (int t = 0; t < P; ++t) {
    i64 re[Q], im[Q];
    phase3<N>(re, im, t, sl.data());
    for (int q = 0; q < Q && t + P * q < n; ++q) {
      for (int l = 0; l < 2; ++l) {
        const double c = line_coef(n == N ? -dk2 * (N / 4) : dk2 * (0.5 * n * n / N), em[l], lb[l], drop);
        out[l * n + t + P * q] = c * bits_double(to_bits(l == 0 ? re[q] : im[q]));
      }
    }
  }
}

extern "C" int fx_line(int n, int m, const double* in, double dk2, double* out) {  // m: transform length
  switch (m) {
    case 16: line<16>(n, in, dk2, out); return 0;
    case 32: line<32>(n, in, dk2, out); return 0;
    case 64: line<64>(n, in, dk2, out); return 0;
    case 128: line<128>(n, in, dk2, out); return 0;
    case 256: line<256>(n, in, dk2, out); return 0;
    case 512: line<512>(n, in, dk2, out); return 0;
    default: return 1;
  }
}
extern "C" double fx_round(long long v) { return bits_double(to_bits(v)); }
