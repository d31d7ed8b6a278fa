// fx.cuh -- one-dimensional spectral second derivatives of FP64 lines in
// 64-bit fixed point.
//
// Why integers: GB300 issues 2 FP64 operations per clock and SM (measured
// 1.6, additions and multiply-adds alike) but 60 64-bit integer additions
// and 60 32 x 32 + 64-bit multiply-adds (mad.wide).  A line transform is
// additions and multiplications by numbers of modulus at most one, so its
// values never outgrow a bound known before it starts, and a fixed-point
// number with one exponent per line carries it: a complex addition costs 4
// issue slots instead of 128, a complex product about 42 instead of 256.
//
// Format.  A real line is shifted by its own first value (the derivative
// does not see a constant) and scaled by a power of two so that the sum of
// its moduli stays below 2^61.  Two real lines A, B form the complex line
// A + iB; each keeps its own exponent, since the real, even multiplier never
// mixes them.  Bounds: every partial sum of the forward transform has parts
// below 2^62; the multiplier h_f = (2 f / N)^2 is at most 1; and because the
// kernel of h has unit l1 norm (its entries alternate in sign and h at the
// Nyquist frequency is 1), every partial sum of the unnormalised inverse is
// below sqrt(2) N times the line's largest value, which the multiplier's
// `drop` bits keep below 2^62.  Nothing overflows and no stage is rescaled.
//
// Error.  The line enters with an absolute rounding of one unit, less than
// N 2^-60 of its largest deviation: 2^-54 to 2^-57 of it on noise, 2^-51 where
// 512 deviations are of one size.  Each product rounds to one unit of the
// growing spectrum, whose relative weight falls with every stage; the FP64
// transform rounds every operation to 2^-53 of its result.  The derivative's
// error stays below 8 2^-53 of the largest that such a line can have
// (tests/test_fx_lines.py).
//
// A product x w with w = W 2^-62: x = xh 2^32 + xl and W = Wh 2^32 + Wl with
// signed low halves, x W 2^-62 = (xh Wh) 4 + (xh Wl + xl Wh) 2^-30 + (xl Wl)
// 2^-62; the last term is below one unit and left out.
#pragma once
#include <type_traits>
#include <utility>

#include "fx_tables.h"

#ifdef __CUDACC__
#define LAT_HD __host__ __device__ __forceinline__
#else  // the host test of the line transforms
#define LAT_HD inline
#endif

namespace lat {
namespace fx {

using i64 = long long;
using u64 = unsigned long long;

struct alignas(16) Cx64 {
  i64 x, y;
};
// a twiddle exp(-2 pi i j / n) as split integers
struct alignas(16) Tw {
  int rh, rl, ih, il;
};

// W = wh 2^32 + wl with wl in [-2^31, 2^31)
constexpr int split_lo(i64 w) { return (int)(unsigned int)(u64)w; }
constexpr int split_hi(i64 w) { return (int)((w - split_lo(w)) / 4294967296LL); }

LAT_HD int lo_of(i64 x) { return (int)(unsigned int)(u64)x; }
LAT_HD int hi_of(i64 x) { return (int)((x + 0x80000000LL) >> 32); }  // x = hi_of 2^32 + lo_of (signed low half)
// a b + c; spelled out for the device, where the compiler splits the sum of
// products into 64-bit multiplications and additions (75 instructions a
// complex product instead of 3x)
LAT_HD i64 mad(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
  i64 d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (i64)a * b + c;
#endif
}
LAT_HD i64 mulw(int a, int b) {
#ifdef __CUDA_ARCH__
  i64 d;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
  return d;
#else
  return (i64)a * b;
#endif
}
LAT_HD i64 shl(i64 x, int n) { return (i64)((u64)x << n); }

// x c for a real constant of modulus <= 1
LAT_HD i64 rmul(i64 x, int ch, int cl) {
  const int h = hi_of(x), l = lo_of(x);
  const i64 mid = mad(h, cl, mad(l, ch, 1LL << 29));
  return shl(mulw(h, ch), 2) + (mid >> 30);
}

// (xr, xi) *= w (CONJ: its conjugate)
template <bool CONJ>
LAT_HD void cmul(i64& xr, i64& xi, const Tw& w) {
  const int rh = hi_of(xr), rl = lo_of(xr), ih = hi_of(xi), il = lo_of(xi);
  // re = xr wr - xi wi, im = xr wi + xi wr (wi of the other sign for CONJ)
  const int sih = CONJ ? w.ih : -w.ih, sil = CONJ ? w.il : -w.il;
  const i64 hr = mad(ih, sih, mulw(rh, w.rh));
  const i64 mr = mad(ih, sil, mad(il, sih, mad(rh, w.rl, mad(rl, w.rh, 1LL << 29))));
  const i64 hi = mad(rh, -sih, mulw(ih, w.rh));
  const i64 mi = mad(rh, -sil, mad(rl, -sih, mad(ih, w.rl, mad(il, w.rh, 1LL << 29))));
  xr = shl(hr, 2) + (mr >> 30);
  xi = shl(hi, 2) + (mi >> 30);
}

// (xr, xi) *= exp(-+ 2 pi i J / 32) (INV: +)
template <int J0, bool INV>
LAT_HD void cmul_const(i64& xr, i64& xi) {
  constexpr int J = ((INV ? 32 - J0 % 32 : J0) % 32 + 32) % 32;
  if constexpr (J == 0) {
    return;
  } else if constexpr (J == 8) {  // -i
    const i64 t = xr;
    xr = xi;
    xi = -t;
  } else if constexpr (J == 16) {
    xr = -xr;
    xi = -xi;
  } else if constexpr (J == 24) {  // i
    const i64 t = xr;
    xr = -xi;
    xi = t;
  } else if constexpr (J % 8 == 4) {
    constexpr int ch = split_hi(kCos32[4]), cl = split_lo(kCos32[4]);
    const i64 s = rmul(xr + xi, ch, cl), d = rmul(xi - xr, ch, cl);  // exp(-i pi/4): (s, d)
    if constexpr (J == 4) { xr = s; xi = d; }
    else if constexpr (J == 12) { xr = d; xi = -s; }   // times -i
    else if constexpr (J == 20) { xr = -s; xi = -d; }
    else { xr = -d; xi = s; }
  } else {
    constexpr i64 c = kCos32[J], s = kCos32[(J + 8) % 32];  // -sin(2 pi J/32) = cos(2 pi (J + 8)/32)
    constexpr Tw w{split_hi(c), split_lo(c), split_hi(s), split_lo(s)};
    cmul<false>(xr, xi, w);
  }
}

template <int... I, typename F>
LAT_HD void static_for_impl(std::integer_sequence<int, I...>, F&& f) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
LAT_HD void static_for(F&& f) {
  static_for_impl(std::make_integer_sequence<int, N>{}, f);
}

// 4-point DFT of four values in place: y0,2 = (a + c) +- (b + d), y1,3 = (a - c) -+ i (b - d)
template <bool INV>
LAT_HD void dft4(i64& ar, i64& ai, i64& br, i64& bi, i64& cr, i64& ci, i64& dr, i64& di) {
  const i64 sr = ar + cr, si = ai + ci, tr = ar - cr, ti = ai - ci;
  const i64 ur = br + dr, ui = bi + di, vr = br - dr, vi = bi - di;
  ar = sr + ur;
  ai = si + ui;
  cr = sr - ur;
  ci = si - ui;
  if (INV) {
    br = tr - vi;
    bi = ti + vr;
    dr = tr + vi;
    di = ti - vr;
  } else {
    br = tr + vi;
    bi = ti - vr;
    dr = tr - vi;
    di = ti + vr;
  }
}

// In-register DFT of R = 2 ... 32 points (a power of two), natural order in and
// out: radix 4 (or 2) by decimation in time.
template <int R, bool INV>
LAT_HD void dft(i64 (&re)[R], i64 (&im)[R]) {
  static_assert(32 % R == 0, "twiddles come from the 32-point table");
  if constexpr (R == 2) {
    const i64 a = re[0], b = im[0];
    re[0] = a + re[1];
    im[0] = b + im[1];
    re[1] = a - re[1];
    im[1] = b - im[1];
  } else if constexpr (R == 4) {
    dft4<INV>(re[0], im[0], re[1], im[1], re[2], im[2], re[3], im[3]);
  } else {
    constexpr int M = R / 4;  // four interleaved subsequences of M points
    i64 sr[4][M], si[4][M];
    static_for<4>([&](auto b) {
      static_for<M>([&](auto k) {
        sr[b.value][k.value] = re[4 * k.value + b.value];
        si[b.value][k.value] = im[4 * k.value + b.value];
      });
      dft<M, INV>(sr[b.value], si[b.value]);
      static_for<M>([&](auto k) {
        cmul_const<(32 / R) * b.value * k.value, INV>(sr[b.value][k.value], si[b.value][k.value]);
      });
    });
    static_for<M>([&](auto kk) {
      constexpr int k = kk.value;
      dft4<INV>(sr[0][k], si[0][k], sr[1][k], si[1][k], sr[2][k], si[2][k], sr[3][k], si[3][k]);
      static_for<4>([&](auto b) {
        re[k + M * b.value] = sr[b.value][k];
        im[k + M * b.value] = si[b.value][k];
      });
    });
  }
}

// ------------------------------------------------------------ conversions
constexpr int kNanExp = 2047;
constexpr u64 kNan = 0x7ff8000000000000ULL;

LAT_HD int exp_of(u64 b) {  // biased exponent, subnormals with the smallest
  const int e = (int)(b >> 52) & 0x7ff;
  return e > 1 ? e : 1;
}
// the value of the FP64 bits b in units of 2^(emax - 1084), emax >= its
// exponent: below 2^62, exact unless it is 2^10 times smaller than 2^emax
LAT_HD i64 from_bits(u64 b, int emax) {
  const int e = (int)(b >> 52) & 0x7ff;
  u64 m = ((b & 0xfffffffffffffULL) | ((u64)(e != 0) << 52)) << 9;
  const int r = emax - (e > 1 ? e : 1);
#ifdef __CUDA_ARCH__
  asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(r));  // shifts past 63 give 0
#else
  m = r < 64 ? m >> r : 0;
#endif
  const i64 s = (i64)b >> 63;
  return ((i64)m ^ s) - s;
}
LAT_HD int clz64(u64 v) {
#ifdef __CUDA_ARCH__
  return __clzll((i64)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}
// leading zeros of a 32-bit word; -1 for zero
LAT_HD int lead0(unsigned int v) {
#ifdef __CUDA_ARCH__
  int r;
  asm("bfind.shiftamt.u32 %0, %1;" : "=r"(r) : "r"(v));
  return r;
#else
  return v ? __builtin_clz(v) : -1;
#endif
}
// v 2^-61 rounded to FP64, |v| < 2^63 (the power keeps a line's coefficient, below, in range)
LAT_HD u64 to_bits(i64 v) {
  const i64 s = v >> 63;
  u64 m = (u64)((v ^ s) - s);
  const unsigned int hi = (unsigned int)(m >> 32), top = hi ? hi : (unsigned int)m;
  const int sh = lead0(top) + (hi ? -1 : 31);   // moves the leading bit to 62
  m = ((m << sh) + 0x200) >> 10;                // 53 bits; a carry moves into the exponent below
  const unsigned int e = top ? (unsigned int)(1023 - sh) << 20 : 0u;  // the leading bit adds one
  return (m + ((u64)e << 32)) | ((u64)s & 0x8000000000000000ULL);
}
// v 2^(e - 61) rounded to FP64, |v| < 2^63; below the normal range 0, above it infinite
LAT_HD u64 to_bits_exp(i64 v, int e) {
  const i64 s = v >> 63;
  u64 m = (u64)((v ^ s) - s);
  const unsigned int hi = (unsigned int)(m >> 32), top = hi ? hi : (unsigned int)m;
  const int sh = lead0(top) + (hi ? -1 : 31);
  m = ((m << sh) + 0x200) >> 10;
  const int ex = 1023 - sh + e;  // the leading bit adds one
  u64 r = m + ((u64)(unsigned int)ex << 52);
  r = ex > 2045 ? 0x7ff0000000000000ULL : r;
  r = (top == 0 || ex < 0) ? 0 : r;
  return r | ((u64)s & 0x8000000000000000ULL);
}
LAT_HD double bits_double(u64 b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((i64)b);
#else
  double d;
  __builtin_memcpy(&d, &b, 8);
  return d;
#endif
}
LAT_HD u64 double_bits(double d) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(d);
#else
  u64 b;
  __builtin_memcpy(&b, &d, 8);
  return b;
#endif
}
// 2^e for any e, as two factors that are each representable
LAT_HD double pow2_times(double c, int e) {
  const int h = e / 2, r = e - h;
  return c * bits_double((u64)(h + 1023) << 52) * bits_double((u64)(r + 1023) << 52);
}

// ------------------------------------------------------------ line geometry
template <int N> struct Split;  // N = P Q: P threads of Q points per line
template <> struct Split<16> { static constexpr int P = 4, Q = 4, LOG = 4; };
template <> struct Split<32> { static constexpr int P = 4, Q = 8, LOG = 5; };
template <> struct Split<64> { static constexpr int P = 8, Q = 8, LOG = 6; };
template <> struct Split<128> { static constexpr int P = 8, Q = 16, LOG = 7; };
template <> struct Split<256> { static constexpr int P = 16, Q = 16, LOG = 8; };
template <> struct Split<512> { static constexpr int P = 16, Q = 32, LOG = 9; };

// Scale of a line from its deviations d: `ored` the bitwise or of |d| (as d ^
// (d >> 63)), `sum` the sum of (|d| >> 9) + 1.  nm bits hold the largest
// deviation, ns bits the sum of all of them.
struct LineBits {
  int nm, ns;
};
template <int N, int LOG = Split<N>::LOG>
LAT_HD LineBits line_bits(u64 ored, u64 sum) {
  const int nm = 64 - clz64(ored), ns = 64 - clz64(sum) + 9, top = nm + LOG;
  return LineBits{nm, ns < top ? ns : top};
}
// deviations scaled so that their sum stays below 2^61
LAT_HD i64 scale_line(i64 d, LineBits b) { return shl(d, 63 - b.nm) >> (2 + b.ns - b.nm); }
// exponent of a scaled line's unit times 2^61 (to_bits_exp); emax the largest
// biased exponent of the line
LAT_HD int emax_unit(int emax, LineBits b) { return emax - 1084 + b.ns; }
// Bits to drop at the multiplier so that N times the largest value of either
// line stays below 2^61.  A line whose sum is close to its largest value (a
// spike) needs up to log2 N; dropping more than four would cost the other
// line accuracy, so such a line is scaled lower instead.
template <int N>
LAT_HD int drop_bits(LineBits& a, LineBits& b) {
  constexpr int LOG = Split<N>::LOG;
  const int ga = LOG - (a.ns - a.nm), gb = LOG - (b.ns - b.nm);
  const int lo = ga < gb ? ga : gb, hi = ga < gb ? gb : ga;
  const int four = hi < 4 ? hi : 4, g = lo > four ? lo : four;
  if (ga > g) a.ns = a.nm + LOG - g;
  if (gb > g) b.ns = b.nm + LOG - g;
  return g;
}
// What a line's numbers after phase 3 (to_bits: in units of 2^61) are
// multiplied by: the pass's -dk^2 (N/4) times the line's unit 2^(emax - 1084 +
// ns + drop), emax the largest biased exponent of the line.  Exactly zero for a constant line, NaN
// for one that holds a NaN or an infinity.
LAT_HD double line_coef(double c, int emax, LineBits b, int drop) {
  if (emax == kNanExp) return bits_double(kNan);
  if (b.nm == 0) return 0.0;
  return pow2_times(c, emax_unit(emax, b) + drop);
}

// The line transform in three phases; a barrier over the line's threads
// stands between them.  sl: the line's scratch [Q][P + 1]; t1[kq][t] =
// W_N^{t kq} and t2[mp][kq] = W_N^{mp kq}.
template <int N>
LAT_HD void phase1(i64 (&re)[Split<N>::Q], i64 (&im)[Split<N>::Q], int t, Cx64* sl, const Tw* t1) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1;
  dft<Q, false>(re, im);
  static_for<Q>([&](auto kq) {
    constexpr int k = kq.value;
    if constexpr (k != 0) cmul<false>(re[k], im[k], t1[k * P + t]);
    sl[k * S + t] = Cx64{re[k], im[k]};
  });
}
// x f^2 2^-sft, sft = 2 log2(N/2) + drop
LAT_HD i64 hmul(i64 x, int f2, int sft, i64 half) {
  const int h = hi_of(x), l = lo_of(x);
  return shl(mulw(h, f2), 32 - sft) + (mad(l, f2, half) >> sft);
}
template <int N>
LAT_HD void phase2(int t, Cx64* sl, const Tw* t2, int drop) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1, G = Q / P;
  static_assert(Q % P == 0, "rows of a line divide over its threads");
  const int sft = 2 * Split<N>::LOG - 2 + drop;
  const i64 half = 1LL << (sft - 1);
  static_for<G>([&](auto gg) {
    const int kq = t + gg.value * P;
    i64 ur[P], ui[P];
    static_for<P>([&](auto tt) {
      const Cx64 z = sl[kq * S + tt.value];
      ur[tt.value] = z.x;
      ui[tt.value] = z.y;
    });
    dft<P, false>(ur, ui);
    static_for<P>([&](auto kp) {
      const int k = kq + Q * kp.value, f = 2 * kp.value < P ? k : N - k, f2 = f * f;
      ur[kp.value] = hmul(ur[kp.value], f2, sft, half);
      ui[kp.value] = hmul(ui[kp.value], f2, sft, half);
    });
    dft<P, true>(ur, ui);
    static_for<P>([&](auto mp) {
      constexpr int m = mp.value;
      if constexpr (m != 0) cmul<true>(ur[m], ui[m], t2[m * Q + kq]);
      sl[kq * S + m] = Cx64{ur[m], ui[m]};
    });
  });
}
// Lines padded with zeros (k_fxg.cuh): the multiplier is a table of numbers
// below 1 (2^-62 units, split; even, entries 0..N/2) and `drop` bits are dropped.
struct alignas(8) Mult {
  int h, l;
};
template <int N>
LAT_HD void phase2_tab(int t, Cx64* sl, const Tw* t2, const Mult* H, int drop) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1, G = Q / P;
  // rounded: a floor's constant offset on all modes would meet at the first point
  const i64 half = drop > 0 ? 1LL << (drop - 1) : 0;
  static_for<G>([&](auto gg) {
    const int kq = t + gg.value * P;
    i64 ur[P], ui[P];
    static_for<P>([&](auto tt) {
      const Cx64 z = sl[kq * S + tt.value];
      ur[tt.value] = z.x;
      ui[tt.value] = z.y;
    });
    dft<P, false>(ur, ui);
    static_for<P>([&](auto kp) {
      const int k = kq + Q * kp.value;
      const Mult h = H[2 * kp.value < P ? k : N - k];
      ur[kp.value] = (rmul(ur[kp.value], h.h, h.l) + half) >> drop;
      ui[kp.value] = (rmul(ui[kp.value], h.h, h.l) + half) >> drop;
    });
    dft<P, true>(ur, ui);
    static_for<P>([&](auto mp) {
      constexpr int m = mp.value;
      if constexpr (m != 0) cmul<true>(ur[m], ui[m], t2[m * Q + kq]);
      sl[kq * S + m] = Cx64{ur[m], ui[m]};
    });
  });
}

// Forward transform only: row kq of the scratch becomes Z[kq + Q kp], kp < P
// (after phase 1 and a barrier; each row belongs to one thread).
template <int N>
LAT_HD void phase2_forward(int t, Cx64* sl) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1, G = Q / P;
  static_for<G>([&](auto gg) {
    const int kq = t + gg.value * P;
    i64 ur[P], ui[P];
    static_for<P>([&](auto tt) {
      const Cx64 z = sl[kq * S + tt.value];
      ur[tt.value] = z.x;
      ui[tt.value] = z.y;
    });
    dft<P, false>(ur, ui);
    static_for<P>([&](auto kp) { sl[kq * S + kp.value] = Cx64{ur[kp.value], ui[kp.value]}; });
  });
}
template <int N>
LAT_HD const Cx64& mode_at(const Cx64* sl, int k) {
  return sl[(k % Split<N>::Q) * (Split<N>::P + 1) + k / Split<N>::Q];
}
template <int N>
LAT_HD void phase3(i64 (&re)[Split<N>::Q], i64 (&im)[Split<N>::Q], int t, const Cx64* sl) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1;
  static_for<Q>([&](auto kq) {
    const Cx64 z = sl[kq.value * S + t];
    re[kq.value] = z.x;
    im[kq.value] = z.y;
  });
  dft<Q, true>(re, im);
}

}  // namespace fx
}  // namespace lat
