// fx_host.hpp -- tables of the fixed-point transforms, made on the host.
#pragma once
#include <cmath>
#include <vector>

#include "fx.cuh"

namespace lat {
namespace fx {

// exp(-2 pi i j / n), j < n, as split integers; n a multiple of 8 (cos and sin
// are evaluated on an eighth of the circle)
inline void roots(int n, Tw* w) {
  std::vector<long long> c(n / 4 + 1);  // cos on the first quadrant, 2^-62 units
  const long double one = 4611686018427387904.0L, step = 6.283185307179586476925286766559L / (long double)n;
  for (int j = 0; j <= n / 8; ++j) {
    c[j] = llrintl(cosl(step * j) * one);
    c[n / 4 - j] = llrintl(sinl(step * j) * one);
  }
  auto cosj = [&](int j) {  // 0 <= j < n
    if (j > n / 2) j = n - j;
    return j <= n / 4 ? c[j] : -c[n / 2 - j];
  };
  for (int j = 0; j < n; ++j) {
    const long long re = cosj(j), im = cosj((j + n / 4) % n);  // -sin(t) = cos(t + pi/2)
    w[j] = Tw{split_hi(re), split_lo(re), split_hi(im), split_lo(im)};
  }
}

// Half the multiplier of a side of n points on lines padded to m (k_fxg.cuh),
// entries 0..m/2 in 2^-62 units: c_0/2 + sum_j c_j cos(2 pi j k / m) with the
// taps c_j of the second derivative over (n/2)^2; w: W_m^j.
inline void multiplier(int n, int m, const Tw* w, Mult* H) {
  const long double pi = 3.141592653589793238462643383280L, one = 4611686018427387904.0L;
  const long double scale = 4.0L / ((long double)n * n);
  std::vector<long long> c(n), co(m);
  const long double c0 = n % 2 ? -((long double)n * n - 1) / 12 : -((long double)n * n + 2) / 12;
  c[0] = llrintl(c0 * scale * one);
  for (int j = 1; j <= n / 2; ++j) {
    const long double sn = sinl(pi * j / n);
    long double v = (j % 2 ? 0.5L : -0.5L) / (sn * sn);
    if (n % 2) v *= cosl(pi * j / n);
    c[j] = llrintl(v * scale * one);
    c[n - j] = c[j];
  }
  for (int j = 0; j < m; ++j) co[j] = (long long)w[j].rh * 4294967296LL + w[j].rl;
  for (int k = 0; k <= m / 2; ++k) {
    __int128 acc = (__int128)c[0] << 61;
    for (int j = 1; j < n; ++j) acc += (__int128)c[j] * co[(int)((long long)j * k % m)];
    const long long v = (long long)((acc + ((__int128)1 << 61)) >> 62);
    H[k] = Mult{split_hi(v), split_lo(v)};
  }
}

}  // namespace fx
}  // namespace lat
