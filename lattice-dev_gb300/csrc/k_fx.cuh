// k_fx.cuh -- separable spectral passes of FP64 lattices with fixed-point
// line transforms (sm_103a).
//
// The passes of a kick (laplacian_3d, Pseudospec/openmp_dev/fftw_mod.f90:
// 177-207, as a sum of three line derivatives; Hamiltonian pieces of
// hamiltonian_conformal.f90:86-174 and hamiltonian_minkowski.f90:86-136):
//
//   X: drift phi, lap  = d2x(phi)                 [+ sum pi^2 of the drift]
//   Y:            lap += d2y(phi)
//   Z: pi += ck (lap + d2z(phi)) - cv V'(phi)     [+ GE2, PE, Friedmann]
//
// all in place: a site is read and written by one thread of one block.  The
// FP64 pipe (2 operations per clock and SM) bounds whatever runs on it, so the
// line transforms run in 64-bit integers (fx.cuh) and FP64 is left to what the
// Hamiltonian itself needs per site: 6 operations in X, 2 in Y and 17 in Z
// (two fields, expanding); conversions are integer operations too, about 190
// instructions per value, line derivative included.  256^3, two fields, per
// pass: X 0.45, Y 0.39, Z 0.72 ms and 4.8 ms a Yoshida-4 step, against 24.8 ms
// with FP64 transforms (3D cuFFT).  X and Y are bound by instruction issue at
// 16 warps an SM (128 registers a thread), Z by the FP64 pipe (76% busy).
//
// Two real lines share one complex transform: the two fields at the same
// sites, or (one field) two neighbouring lines.  A block takes 16 complex
// lines and loops over tiles; P threads hold Q = N / P points of a line each.
#pragma once
#include <algorithm>

#include "engine.hpp"
#include "fx.cuh"

namespace lat {
namespace fx {

constexpr int kLines = 16;  // complex lines of a tile

template <int N>
struct Geo {
  static constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1;
  static constexpr int THREADS = kLines * P;
  static constexpr int LSTRIDE = (Q * S) | 1;  // odd: the lines of a quarter warp start in different banks
  static constexpr int SMEM = (2 * N + kLines * LSTRIDE) * 16;
  // 128 registers a thread (512 points: 32 complex values a thread, 255)
  static constexpr int MINB = N == 512 ? 1 : (THREADS == 256 ? 2 : (THREADS == 128 ? 4 : 6));
};

// sites of complex line l: the two real lines' first sites and the stride
template <int AXIS, int NF>
__device__ __forceinline__ void line_at(int64_t l, int nx, int ny, int64_t Ns, int64_t& a, int64_t& b, int64_t& st) {
  if (AXIS == 0) {
    st = 1;
    a = NF == 2 ? l * nx : 2 * l * nx;
    b = NF == 2 ? Ns + a : a + nx;
  } else {
    const int64_t plane = (int64_t)nx * ny;
    st = AXIS == 1 ? nx : plane;
    const int per = NF == 2 ? nx : nx / 2;
    const int64_t o = l / per;
    const int x = (int)(l - o * per) * (NF == 2 ? 1 : 2);
    a = (AXIS == 1 ? o * plane : o * nx) + x;
    b = NF == 2 ? Ns + a : a + 1;
  }
}

// the two lines' values at one position: one 16-byte access where they are neighbours
template <int AXIS, int NF>
__device__ __forceinline__ double2 ld2(const double* p, int64_t a, int64_t b) {
  if (NF == 1 && AXIS != 0) return *reinterpret_cast<const double2*>(p + a);
  return make_double2(p[a], p[b]);
}
template <int AXIS, int NF>
__device__ __forceinline__ void st2(double* p, int64_t a, int64_t b, double2 v) {
  if (NF == 1 && AXIS != 0) {
    *reinterpret_cast<double2*>(p + a) = v;
  } else {
    p[a] = v.x;
    p[b] = v.y;
  }
}

// Line-wide maximum, or and sum.  Pass X keeps a line inside P neighbouring
// lanes; in Y and Z a warp holds two threads of each of the 16 lines, and the
// warps meet in shared memory (W = P / 2 rows of 16 lines).
template <int AXIS, int P, typename T, typename F>
__device__ __forceinline__ T line_reduce(T v, F op, T (*sh)[kLines], int li, int warp) {
  if constexpr (AXIS == 0) {
#pragma unroll
    for (int o = 1; o < P; o <<= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  } else {
    v = op(v, __shfl_xor_sync(0xffffffffu, v, kLines));
    sh[warp][li] = v;  // both lanes write the same value
    return v;
  }
}
template <int AXIS, int P, typename T, typename F>
__device__ __forceinline__ T line_collect(T v, F op, T (*sh)[kLines], int li) {
  if constexpr (AXIS != 0) {
    v = sh[0][li];
#pragma unroll
    for (int w = 1; w < P / 2; ++w) v = op(v, sh[w][li]);
  }
  return v;
}
template <int AXIS>
__device__ __forceinline__ void line_barrier() {
  if constexpr (AXIS == 0) __syncwarp();
  else __syncthreads();
}

// V' at one site and the site's term of 4 V (2 V for the free model), in as
// few FP64 operations as the model allows: 7 + 2 for the coupled quartic one.
template <int MODEL, int NF>
__device__ __forceinline__ void force(double p0, double p1, double2 f, double2& dv, double& v4) {
  if constexpr (MODEL == LAT_MODEL_PHI4_G2 && NF == 2) {
    const double x2 = f.x * f.x, y2 = f.y * f.y;
    dv.x = f.x * fma(p1, y2, p0 * x2);
    dv.y = (p1 * x2) * f.y;
    v4 = fma(f.y, dv.y, fma(f.x, dv.x, v4));
  } else if constexpr (MODEL == LAT_MODEL_DOUBLE_WELL) {
    const double tx = fma(f.x, f.x, -1.0);
    dv.x = fma(tx, f.x, -p0);
    v4 = fma(tx, tx, v4) - 4.0 * p0 * (f.x + 1.0);
    if (NF == 1) {
      const double ty = fma(f.y, f.y, -1.0);
      dv.y = fma(ty, f.y, -p0);
      v4 = fma(ty, ty, v4) - 4.0 * p0 * (f.y + 1.0);
    } else {
      dv.y = 0.0;
    }
  } else if constexpr (MODEL == LAT_MODEL_FREE) {
    dv.x = p0 * f.x;
    dv.y = p0 * f.y;
    v4 = fma(f.y, dv.y, fma(f.x, dv.x, v4));
  } else {  // quartic; a second field is free of forces
    dv.x = p0 * (f.x * f.x) * f.x;
    v4 = fma(f.x, dv.x, v4);
    if (NF == 1) {
      dv.y = p0 * (f.y * f.y) * f.y;
      v4 = fma(f.y, dv.y, v4);
    } else {
      dv.y = 0.0;
    }
  }
}

// The kick of pass Z at the thread's Q sites, whose line derivatives (as
// integers) wait in the thread's own scratch places.
template <int MODEL, int NF, int N, bool CONF>
__device__ __forceinline__ void kick_sites(const ModelP& m, const double* __restrict__ phi, double* pi,
                                           const double* __restrict__ lap, const Cx64* sl, int t, int64_t oa,
                                           int64_t ob, int64_t st, double ca, double cb, double ck, double cv,
                                           double& ge, double& pe) {
  constexpr int P = Split<N>::P, Q = Split<N>::Q, S = P + 1;
  const double p0 = m.p[0], p1 = m.p[1];
  double v4 = 0.0;
#pragma unroll 4
  for (int q = 0; q < Q; ++q) {
    const int64_t o = (t + P * q) * st;
    const Cx64 z = sl[q * S + t];
    const double2 b = ld2<2, NF>(lap, oa + o, ob + o), f = ld2<2, NF>(phi, oa + o, ob + o);
    double2 p = ld2<2, NF>(pi, oa + o, ob + o), dv;
    const double lx = fma(ca, bits_double(to_bits(z.x)), b.x),
                 ly = fma(cb, bits_double(to_bits(z.y)), b.y);
    force<MODEL, NF>(p0, p1, f, dv, v4);
    p.x = fma(-cv, dv.x, fma(ck, lx, p.x));
    p.y = fma(-cv, dv.y, fma(ck, ly, p.y));
    st2<2, NF>(pi, oa + o, ob + o, p);
    if (CONF) ge = fma(-f.y, ly, fma(-f.x, lx, ge));
  }
  if (CONF) pe = fma(MODEL == LAT_MODEL_FREE ? 0.5 : 0.25, v4, pe);
}

// The lines of a tile of one array into L2, 128 bytes per request.
template <int NF, int AXIS, int N>
__device__ __forceinline__ void prefetch_tile(const double* p, int64_t tile, int nx, int ny, int64_t Ns, int tid) {
  int64_t a, b, st;
  line_at<AXIS, NF>(tile * kLines, nx, ny, Ns, a, b, st);
  for (int i = tid; i < 2 * N; i += Geo<N>::THREADS) {
    int64_t o;
    if (NF == 2) o = (i < N ? a : b) + (AXIS == 0 ? 16 * (i % N) : (i % N) * st);
    else o = a + (AXIS == 0 ? 16 * i : (i >> 1) * st + 16 * (i & 1));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
  }
}

template <int NF, int AXIS, int N, bool CONF>
__global__ void __launch_bounds__(Geo<N>::THREADS, Geo<N>::MINB) fx_kernel(SepArgs a) {
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
  const Tw* tw = static_cast<const Tw*>(a.twN);  // W_N^j
  for (int i = tid; i < N; i += G::THREADS) {
    t1[i] = tw[((i / P) * (i % P)) % N];
    t2[i] = tw[((i / Q) * (i % Q)) % N];
  }
  // the coefficients once per block (their divisions would load the FP64 pipe)
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
  const int64_t Ns = (int64_t)a.nx * a.ny * a.nz;
  double* phi = static_cast<double*>(a.phi_out);
  double* pi = static_cast<double*>(a.pi_out);
  double* lap = static_cast<double*>(a.lap_out);
  const double cline = -a.dk2 * (N / 4);
  const bool drift = AXIS == 0 && a.hd != 0.0;
  double ke = 0.0, pe = 0.0, ge = 0.0;
  bool nonfinite = false;
  auto imax = [](int x, int y) { return max(x, y); };
  auto oor = [](u64 x, u64 y) { return x | y; };
  auto add = [](u64 x, u64 y) { return x + y; };

  const int64_t ntile = a.nlines / kLines;  // whole tiles: sides are powers of two from 16 on
  for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    int64_t oa, ob, st;
    line_at<AXIS, NF>(tile * kLines + li, a.nx, a.ny, Ns, oa, ob, st);
    // the values wait in the thread's own scratch places between the steps, so
    // that all but the transform itself are short loops: unrolled over the
    // thread's points the pass outgrew the instruction cache
    int ea = 1, eb = 1;
#pragma unroll 8
    for (int q = 0; q < Q; ++q) {
      const int64_t o = (t + P * q) * st;
      double2 f = ld2<AXIS, NF>(phi, oa + o, ob + o);
      if (drift) {
        const double2 p = ld2<AXIS, NF>(pi, oa + o, ob + o);
        f.x = fma(cd, p.x, f.x);
        f.y = fma(cd, p.y, f.y);
        if (CONF) ke = fma(p.y, p.y, fma(p.x, p.x, ke));
        st2<AXIS, NF>(phi, oa + o, ob + o, f);
      }
      const u64 ba = double_bits(f.x), bb = double_bits(f.y);
      ea = max(ea, exp_of(ba));
      eb = max(eb, exp_of(bb));
      sl[q * G::S + t] = Cx64{(i64)ba, (i64)bb};
    }
    if (tile + gridDim.x < ntile) {  // what the block's next tile will load
      const int64_t nt = tile + gridDim.x;
      prefetch_tile<NF, AXIS, N>(phi, nt, a.nx, a.ny, Ns, tid);
      if (drift || AXIS == 2) prefetch_tile<NF, AXIS, N>(pi, nt, a.nx, a.ny, Ns, tid);
      if (AXIS != 0) prefetch_tile<NF, AXIS, N>(lap, nt, a.nx, a.ny, Ns, tid);
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
    u64 oA = 0, oB = 0, sA = 0, sB = 0;
#pragma unroll 4
    for (int q = 0; q < Q; ++q) {
      Cx64 z = sl[q * G::S + t];
      z.x = from_bits((u64)z.x, ea) - xa;
      z.y = from_bits((u64)z.y, eb) - xb;
      sl[q * G::S + t] = z;
      const u64 ma = (u64)(z.x ^ (z.x >> 63)), mb = (u64)(z.y ^ (z.y >> 63));
      oA |= ma;
      oB |= mb;
      sA += ma >> 9;
      sB += mb >> 9;
    }
    sA += Q;
    sB += Q;
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
    phase2<N>(t, sl, t2, drop);
    line_barrier<AXIS>();
    phase3<N>(re, im, t, sl);
    const double ca = line_coef(cline, ea, ba, drop), cb = line_coef(cline, eb, bb, drop);
    nonfinite = nonfinite || ea == kNanExp || eb == kNanExp;
#pragma unroll
    for (int q = 0; q < Q; ++q) sl[q * G::S + t] = Cx64{re[q], im[q]};
    if constexpr (AXIS == 2) {
      switch (a.model.model) {
        case LAT_MODEL_PHI4:
          kick_sites<LAT_MODEL_PHI4, NF, N, CONF>(a.model, phi, pi, lap, sl, t, oa, ob, st, ca, cb, ck, cv, ge, pe);
          break;
        case LAT_MODEL_PHI4_G2:
          kick_sites<LAT_MODEL_PHI4_G2, NF, N, CONF>(a.model, phi, pi, lap, sl, t, oa, ob, st, ca, cb, ck, cv, ge, pe);
          break;
        case LAT_MODEL_DOUBLE_WELL:
          kick_sites<LAT_MODEL_DOUBLE_WELL, NF, N, CONF>(a.model, phi, pi, lap, sl, t, oa, ob, st, ca, cb, ck, cv, ge,
                                                         pe);
          break;
        default:
          kick_sites<LAT_MODEL_FREE, NF, N, CONF>(a.model, phi, pi, lap, sl, t, oa, ob, st, ca, cb, ck, cv, ge, pe);
      }
    } else {
#pragma unroll 8
      for (int q = 0; q < Q; ++q) {
        const int64_t o = (t + P * q) * st;
        const Cx64 z = sl[q * G::S + t];
        double2 d = make_double2(bits_double(to_bits(z.x)), bits_double(to_bits(z.y)));
        if (AXIS == 0) {
          d.x *= ca;
          d.y *= cb;
        } else {
          const double2 b = ld2<AXIS, NF>(lap, oa + o, ob + o);
          d.x = fma(ca, d.x, b.x);
          d.y = fma(cb, d.y, b.y);
        }
        st2<AXIS, NF>(lap, oa + o, ob + o, d);
      }
    }
    // Y, Z: the next tile writes emx and first after this tile's last two
    // barriers, behind every read of them, and ors and sums likewise.  A
    // thread's scratch places are its own outside phase 2, which two barriers
    // enclose.
    if constexpr (AXIS == 0) __syncwarp();
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
int fx_go(const SepArgs& a, cudaStream_t s) {
  using G = Geo<N>;
  auto k = fx_kernel<NF, AXIS, N, CONF>;
  // also below 48 KB, which the static arrays count towards
  const cudaError_t ea = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
  if (ea != cudaSuccess) return cuda_fail(ea, "fixed-point pass smem attribute");
  const int64_t tiles = a.nlines / kLines;
  if (a.nlines % kLines) return set_error(LAT_ERR_STATE, "fixed-point pass: partial tile");
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)a.nsm * G::MINB);
  k<<<grid, G::THREADS, G::SMEM, s>>>(a);
  if (g_launch_counter) ++*g_launch_counter;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, "fixed-point pass launch");
}

template <int N>
int fx_dispatch(const SepArgs& a, int axis, cudaStream_t s) {
#define LAT_FX_AX(NF, CF)                                \
  switch (axis) {                                        \
    case 0: return fx_go<NF, 0, N, CF>(a, s);            \
    case 1: return fx_go<NF, 1, N, false>(a, s);         \
    default: return fx_go<NF, 2, N, CF>(a, s);           \
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
