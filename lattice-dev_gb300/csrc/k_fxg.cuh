// k_fxg.cuh -- fixed-point spectral passes of FP64 lattices for sides that are
// no power of two (sm_103a).
//
// The derivative along a line of n points is a circular sum with the kernel
// c_j = -(-1)^j / (2 sin^2(pi j / n)) (n even; times cos(pi j / n) for odd n),
// c_0 = -(n^2 + 2) / 12 (odd: -(n^2 - 1) / 12), in units of dk^2: the inverse
// transform of laplacian_3d's -f^2 (Pseudospec/openmp_dev/fftw_mod.f90:
// 192-201).  Any length M >= 2 n - 1 can carry it: the line padded with zeros
// to M points, transformed, multiplied by the (real, even) transform H of the
// kernel laid out on -(n-1)..(n-1), and transformed back holds the derivative
// in its first n points.  So sides up to 256 run the power-of-two transforms
// of fx.cuh with M = 64 ... 512 and a table H, at two to four times the work of
// a direct transform, which still beats cuFFT's FP64 transforms of n points. A
// kick of one field: 150 x 108 x 96 200 us against 456, 192^3 1.1 ms against
// 1.8, 127 x 131 x 113 (cuFFT pads primes too) 0.22 ms against 2.0.
//
// Bounds: the taps divided by (n/2)^2 have l1 norm at most 1 on the circle of n
// points, so at most 2 on the padded line; H enters halved, and the values
// obey the bounds of the power-of-two passes.
//
// Lines are numbered through (o, x); a tile takes 16 complex lines, the last
// one what is left, and with one field the lines 2 l and 2 l + 1.
#pragma once
#include "k_fx.cuh"

namespace lat {
namespace fx {

// first site and stride of real line l
template <int AXIS>
__device__ __forceinline__ int64_t line_base(int64_t l, int nx, int ny) {
  if (AXIS == 0) return l * nx;
  if (AXIS == 1) return (l / nx) * ((int64_t)nx * ny) + l % nx;
  return l;
}

template <int MODEL, int NF, int N, bool CONF>
__device__ __forceinline__ void kick_sites_any(const ModelP& m, const double* __restrict__ phi, double* pi,
                                               const double* __restrict__ lap, const Cx64* sl, int t, int n,
                                               int64_t oa, int64_t ob, bool vb, int64_t st, double ca, double cb,
                                               double ck, double cv, double& ge, double& pe) {
  constexpr int P = Split<N>::P, S = P + 1;
  const double p0 = m.p[0], p1 = m.p[1];
  double v4 = 0.0;
#pragma unroll 4
  for (int i = t; i < n; i += P) {
    const int64_t a = oa + i * st, b = vb ? ob + i * st : a;  // without a second line the first one twice
    const Cx64 z = sl[(i / P) * S + t];
    const double2 f = make_double2(phi[a], phi[b]), l0 = make_double2(lap[a], lap[b]);
    double2 p = make_double2(pi[a], pi[b]), dv;
    const double lx = fma(ca, bits_double(to_bits(z.x)), l0.x), ly = fma(cb, bits_double(to_bits(z.y)), l0.y);
    double w = 0.0;
    force<MODEL, NF>(p0, p1, f, dv, w);
    p.x = fma(-cv, dv.x, fma(ck, lx, p.x));
    p.y = fma(-cv, dv.y, fma(ck, ly, p.y));
    pi[a] = p.x;
    if (vb) pi[b] = p.y;
    if (CONF) {
      v4 += NF == 1 && !vb ? 0.5 * w : w;
      ge = fma(-f.x, lx, ge);
      if (vb) ge = fma(-f.y, ly, ge);
    }
  }
  if (CONF) pe = fma(MODEL == LAT_MODEL_FREE ? 0.5 : 0.25, v4, pe);
}

template <int NF, int AXIS, int N, bool CONF>
__global__ void __launch_bounds__(Geo<N>::THREADS, Geo<N>::MINB) fxg_kernel(SepArgs a) {
  using G = Geo<N>;
  constexpr int P = G::P, Q = G::Q, W = P / 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  Tw* t1 = reinterpret_cast<Tw*>(smraw);
  Tw* t2 = t1 + N;
  Cx64* scratch = reinterpret_cast<Cx64*>(t2 + N);
  __shared__ int emx[2][W][kLines];
  __shared__ u64 ors[2][W][kLines], sums[2][W][kLines], first[2][kLines];
  __shared__ double coef_sh[4];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int t = AXIS == 0 ? tid % P : tid / kLines;
  const int li = AXIS == 0 ? tid / P : tid % kLines;
  Cx64* sl = scratch + li * G::LSTRIDE;
  const Tw* tw = static_cast<const Tw*>(a.twN);  // W_N^j, then H
  const Mult* H = reinterpret_cast<const Mult*>(tw + N);
  for (int i = tid; i < N; i += G::THREADS) {
    t1[i] = tw[((i / P) * (i % P)) % N];
    t2[i] = tw[((i / Q) * (i % Q)) % N];
  }
  if (tid == 0) {
    double c0 = a.hd, c1 = a.hk, c2 = a.hk, c3 = 1.0;
    if (CONF) {
      const double a0 = __ldcg(&a.sc->a);
      if (AXIS == 0) {
        c0 = a.hd / (a0 * a0);
      } else if (AXIS == 2) {
        const double a1 = a0 - a.hg * __ldcg(&a.sc->ap) / 6.0;  // Hamiltonian_grav_kinetic before the kick
        c1 = a.hk * a1 * a1;
        c2 = a.hk * a1 * a1 * a1 * a1;
        c3 = a1;
      }
    }
    coef_sh[0] = c0;
    coef_sh[1] = c1;
    coef_sh[2] = c2;
    coef_sh[3] = c3;
  }
  __syncthreads();
  const double cd = coef_sh[0], ck = coef_sh[1], cv = coef_sh[2];
  const int n = AXIS == 0 ? a.nx : (AXIS == 1 ? a.ny : a.nz);
  const int64_t Ns = (int64_t)a.nx * a.ny * a.nz, plane = (int64_t)a.nx * a.ny;
  const int64_t st = AXIS == 0 ? 1 : (AXIS == 1 ? a.nx : plane), real_lines = Ns / n;
  double* phi = static_cast<double*>(a.phi_out);
  double* pi = static_cast<double*>(a.pi_out);
  double* lap = static_cast<double*>(a.lap_out);
  const double cline = a.dk2 * (0.5 * n * n / N);
  const bool drift = AXIS == 0 && a.hd != 0.0;
  double ke = 0.0, pe = 0.0, ge = 0.0;
  bool nonfinite = false;
  auto imax = [](int x, int y) { return max(x, y); };
  auto oor = [](u64 x, u64 y) { return x | y; };
  auto add = [](u64 x, u64 y) { return x + y; };

  const int64_t ntile = (a.nlines + kLines - 1) / kLines;
  for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int64_t l = tile * kLines + li;
    const bool va = l < a.nlines, vb = va && (NF == 2 || 2 * l + 1 < real_lines);
    const int64_t oa = va ? line_base<AXIS>(NF == 2 ? l : 2 * l, a.nx, a.ny) : 0;
    const int64_t ob = vb ? (NF == 2 ? Ns + oa : line_base<AXIS>(2 * l + 1, a.nx, a.ny)) : 0;
    int ea = 1, eb = 1;
#pragma unroll 8
    for (int q = 0; q < Q; ++q) {
      const int i = t + P * q;
      u64 ba = 0, bb = 0;
      if (va && i < n) {
        const int64_t sa = oa + i * st, sb = ob + i * st;
        double2 f = make_double2(phi[sa], vb ? phi[sb] : 0.0);
        if (drift) {
          const double2 p = make_double2(pi[sa], vb ? pi[sb] : 0.0);
          f.x = fma(cd, p.x, f.x);
          f.y = fma(cd, p.y, f.y);
          if (CONF) ke = fma(p.y, p.y, fma(p.x, p.x, ke));
          phi[sa] = f.x;
          if (vb) phi[sb] = f.y;
        }
        ba = double_bits(f.x);
        bb = double_bits(f.y);
      }
      ea = max(ea, exp_of(ba));
      eb = max(eb, exp_of(bb));
      sl[q * G::S + t] = Cx64{(i64)ba, (i64)bb};
    }
    ea = line_reduce<AXIS, P>(ea, imax, emx[0], li, warp);
    eb = line_reduce<AXIS, P>(eb, imax, emx[1], li, warp);
    u64 fa = (u64)sl[t].x, fb = (u64)sl[t].y;  // thread 0: the line's first value
    if constexpr (AXIS == 0) {
      fa = __shfl_sync(0xffffffffu, fa, 0, P);
      fb = __shfl_sync(0xffffffffu, fb, 0, P);
    } else {
      if (t == 0) {
        first[0][li] = fa;
        first[1][li] = fb;
      }
      __syncthreads();
      fa = first[0][li];
      fb = first[1][li];
    }
    ea = line_collect<AXIS, P>(ea, imax, emx[0], li);
    eb = line_collect<AXIS, P>(eb, imax, emx[1], li);
    const i64 xa = from_bits(fa, ea), xb = from_bits(fb, eb);
    u64 oA = 0, oB = 0, sA = Q, sB = Q;
#pragma unroll 4
    for (int q = 0; q < Q; ++q) {
      Cx64 z = sl[q * G::S + t];
      const bool in = t + P * q < n;
      z.x = in ? from_bits((u64)z.x, ea) - xa : 0;
      z.y = in ? from_bits((u64)z.y, eb) - xb : 0;
      sl[q * G::S + t] = z;
      const u64 ma = (u64)(z.x ^ (z.x >> 63)), mb = (u64)(z.y ^ (z.y >> 63));
      oA |= ma;
      oB |= mb;
      sA += ma >> 9;
      sB += mb >> 9;
    }
    oA = line_reduce<AXIS, P>(oA, oor, ors[0], li, warp);
    oB = line_reduce<AXIS, P>(oB, oor, ors[1], li, warp);
    sA = line_reduce<AXIS, P>(sA, add, sums[0], li, warp);
    sB = line_reduce<AXIS, P>(sB, add, sums[1], li, warp);
    if constexpr (AXIS != 0) __syncthreads();
    oA = line_collect<AXIS, P>(oA, oor, ors[0], li);
    oB = line_collect<AXIS, P>(oB, oor, ors[1], li);
    sA = line_collect<AXIS, P>(sA, add, sums[0], li);
    sB = line_collect<AXIS, P>(sB, add, sums[1], li);
    LineBits ba = line_bits<N>(oA, sA), bb = line_bits<N>(oB, sB);
    const int drop = drop_bits<N>(ba, bb);
    i64 re[Q], im[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const Cx64 z = sl[q * G::S + t];
      re[q] = scale_line(z.x, ba);
      im[q] = scale_line(z.y, bb);
    }
    phase1<N>(re, im, t, sl, t1);
    line_barrier<AXIS>();
    phase2_tab<N>(t, sl, t2, H, drop);
    line_barrier<AXIS>();
    phase3<N>(re, im, t, sl);
    const double ca = line_coef(cline, ea, ba, drop), cb = line_coef(cline, eb, bb, drop);
    nonfinite = nonfinite || ea == kNanExp || eb == kNanExp;
#pragma unroll
    for (int q = 0; q < Q; ++q) sl[q * G::S + t] = Cx64{re[q], im[q]};
    if constexpr (AXIS == 2) {
      const int nv = va ? n : 0;
      switch (a.model.model) {
        case LAT_MODEL_PHI4:
          kick_sites_any<LAT_MODEL_PHI4, NF, N, CONF>(a.model, phi, pi, lap, sl, t, nv, oa, ob, vb, st, ca, cb, ck, cv,
                                                      ge, pe);
          break;
        case LAT_MODEL_PHI4_G2:
          kick_sites_any<LAT_MODEL_PHI4_G2, NF, N, CONF>(a.model, phi, pi, lap, sl, t, nv, oa, ob, vb, st, ca, cb, ck,
                                                         cv, ge, pe);
          break;
        case LAT_MODEL_DOUBLE_WELL:
          kick_sites_any<LAT_MODEL_DOUBLE_WELL, NF, N, CONF>(a.model, phi, pi, lap, sl, t, nv, oa, ob, vb, st, ca, cb,
                                                             ck, cv, ge, pe);
          break;
        default:
          kick_sites_any<LAT_MODEL_FREE, NF, N, CONF>(a.model, phi, pi, lap, sl, t, nv, oa, ob, vb, st, ca, cb, ck, cv,
                                                      ge, pe);
      }
    } else if (va) {
#pragma unroll 8
      for (int q = 0; q < Q; ++q) {
        const int i = t + P * q;
        if (i < n) {
          const int64_t sa = oa + i * st, sb = ob + i * st;
          const Cx64 z = sl[q * G::S + t];
          const double dx = bits_double(to_bits(z.x)), dy = bits_double(to_bits(z.y));
          if (AXIS == 0) {
            lap[sa] = ca * dx;
            if (vb) lap[sb] = cb * dy;
          } else {
            lap[sa] = fma(ca, dx, lap[sa]);
            if (vb) lap[sb] = fma(cb, dy, lap[sb]);
          }
        }
      }
    }
    if constexpr (AXIS == 0) __syncwarp();  // the barriers of the next tile do as in fx_kernel
  }
  if (a.nan_flag && nonfinite) atomicOr(&a.sc->err, 1u);
  if (CONF && AXIS == 0) {
    const double v[1] = {ke};
    double tot[1];
    if (grid_reduce<1>(v, a.rb, tot)) {
      DevScalars* w = a.sc;
      const double a0 = w->a;
      w->ap = w->ap + a.hd * (tot[0] / a.Nd) / (a0 * a0 * a0);  // Hamiltonian_fields_kin
      if (drift) w->ke2 = tot[0];
      if (bad(tot[0])) w->err |= 1u;
    }
  }
  if (CONF && AXIS == 2) {
    const double v[2] = {ge, pe};
    double tot[2];
    if (grid_reduce<2>(v, a.rb, tot)) {
      DevScalars* w = a.sc;
      const double a1 = coef_sh[3];
      const double GE2 = tot[0] / (a1 * a1) / a.Nd, PE = tot[1] / a.Nd;
      const double ap1 = w->ap - a1 * a1 * a1 * (GE2 + 4.0 * PE) * a.hk;  // the kick's ysclp update
      w->pe = PE;
      w->ap = ap1;
      w->a = a1 - a.hg * ap1 / 6.0;  // second Hamiltonian_grav_kinetic
      if (bad(GE2) || bad(PE)) w->err |= 1u;
    }
  }
}

template <int NF, int AXIS, int N, bool CONF>
int fxg_go(const SepArgs& a, cudaStream_t s) {
  using G = Geo<N>;
  auto k = fxg_kernel<NF, AXIS, N, CONF>;
  const cudaError_t ea = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
  if (ea != cudaSuccess) return cuda_fail(ea, "fixed-point pass smem attribute");
  const int64_t tiles = (a.nlines + kLines - 1) / kLines;
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)a.nsm * G::MINB);
  k<<<grid, G::THREADS, G::SMEM, s>>>(a);
  if (g_launch_counter) ++*g_launch_counter;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, "fixed-point pass launch");
}

template <int N>
int fxg_dispatch(const SepArgs& a, int axis, cudaStream_t s) {
#define LAT_FX_AX(NF, CF)                                 \
  switch (axis) {                                         \
    case 0: return fxg_go<NF, 0, N, CF>(a, s);            \
    case 1: return fxg_go<NF, 1, N, false>(a, s);         \
    default: return fxg_go<NF, 2, N, CF>(a, s);           \
  }
  if (a.nf == 2) {
    if (a.conf) { LAT_FX_AX(2, true) }
    LAT_FX_AX(2, false)
  }
  if (a.conf) { LAT_FX_AX(1, true) }
  LAT_FX_AX(1, false)
#undef LAT_FX_AX
}

}  // namespace fx
}  // namespace lat
