// k_fxr.cuh -- 3D real-to-complex transform of FP64 data in fixed point
// (sm_103a): the unnormalised forward DFT of one lattice array as the output
// routines bin it (spectrum_3d, Pseudospec/openmp_dev/analysis_spec.f90:59-102;
// the Parseval sum of the gradient energy), [z][y][nx/2+1] complex FP64.
//
// A 3D FP64 transform by cuFFT runs on GB300's FP64 pipe (2 operations per
// clock and SM): 1.76 ms at 256^3.  Here the lines are transformed in 64-bit
// integers with one exponent per line (fx.cuh), three passes of 16, 16 and 16
// bytes per site:
//   X: pairs of real rows as one complex line, split into their half spectra;
//      FP32-Kahan fields enter as phi_hi - c
//   Y, Z: complex lines in place.
// Bound by instruction issue, as the passes of k_fx.cuh.
#pragma once
#include "k_fx.cuh"

namespace lat {
namespace fx {

struct RowIn {
  const void* hi;   // double, or float with its compensation c (null: none)
  const float* c;
};

template <bool F32>
__device__ __forceinline__ double row_value(const RowIn& in, int64_t i) {
  if constexpr (F32) {
    const double h = widen(__ldg(static_cast<const float*>(in.hi) + i));
    return in.c ? h - widen(__ldg(in.c + i)) : h;
  } else {
    return __ldg(static_cast<const double*>(in.hi) + i);
  }
}

template <int N>
__device__ __forceinline__ void load_twiddles(const Tw* tw, Tw* t1, int tid) {
  constexpr int P = Split<N>::P;
  for (int i = tid; i < N; i += Geo<N>::THREADS) t1[i] = tw[((i / P) * (i % P)) % N];
}

// Rows: complex line l is rows 2 l and 2 l + 1; P lanes of a warp hold one line.
template <int N, bool F32>
__global__ void __launch_bounds__(Geo<N>::THREADS, Geo<N>::MINB) fxr_rows(RowIn in, double2* F, int64_t nlines,
                                                                          const Tw* tw) {
  using G = Geo<N>;
  constexpr int P = G::P, Q = G::Q, HX = N / 2 + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  Tw* t1 = reinterpret_cast<Tw*>(smraw);
  Cx64* scratch = reinterpret_cast<Cx64*>(t1 + N);
  const int tid = threadIdx.x, t = tid % P, li = tid / P;
  Cx64* sl = scratch + li * G::LSTRIDE;
  load_twiddles<N>(tw, t1, tid);
  __syncthreads();
  auto imax = [](int x, int y) { return max(x, y); };
  auto oor = [](u64 x, u64 y) { return x | y; };
  auto add = [](u64 x, u64 y) { return x + y; };
  auto lines = [](auto v, auto op) {  // over the P lanes of the line
#pragma unroll
    for (int o = 1; o < P; o <<= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  };
  const int64_t ntile = nlines / kLines;
  for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int64_t l = tile * kLines + li, a = 2 * l * N, b = a + N;
    int ea = 1, eb = 1;
#pragma unroll 8
    for (int q = 0; q < Q; ++q) {
      const int o = t + P * q;
      const u64 ba = double_bits(row_value<F32>(in, a + o)), bb = double_bits(row_value<F32>(in, b + o));
      ea = max(ea, exp_of(ba));
      eb = max(eb, exp_of(bb));
      sl[q * G::S + t] = Cx64{(i64)ba, (i64)bb};
    }
    ea = lines(ea, imax);
    eb = lines(eb, imax);
    const u64 fa = __shfl_sync(0xffffffffu, (u64)sl[t].x, 0, P), fb = __shfl_sync(0xffffffffu, (u64)sl[t].y, 0, P);
    const i64 xa = from_bits(fa, ea), xb = from_bits(fb, eb);
    u64 oA = 0, oB = 0, sA = Q, sB = Q;
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
    oA = lines(oA, oor);
    oB = lines(oB, oor);
    sA = lines(sA, add);
    sB = lines(sB, add);
    const LineBits ba = line_bits<N>(oA, sA), bb = line_bits<N>(oB, sB);
    i64 re[Q], im[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const Cx64 z = sl[q * G::S + t];
      re[q] = scale_line(z.x, ba);
      im[q] = scale_line(z.y, bb);
    }
    phase1<N>(re, im, t, sl, t1);
    __syncwarp();
    phase2_forward<N>(t, sl);
    __syncwarp();
    // the two rows' half spectra: (Z_k + conj Z_{N-k}) / 2 and (Z_k - conj Z_{N-k}) / 2i
    const int ua = emax_unit(ea, ba) - 1, ub = emax_unit(eb, bb) - 1;
    double2* Fa = F + 2 * l * HX;
    for (int k = t; k < HX; k += P) {
      const Cx64 z = mode_at<N>(sl, k), w = mode_at<N>(sl, (N - k) % N);
      double2 A = make_double2(bits_double(to_bits_exp(z.x + w.x, ua)), bits_double(to_bits_exp(z.y - w.y, ua)));
      double2 B = make_double2(bits_double(to_bits_exp(z.y + w.y, ub)), bits_double(to_bits_exp(w.x - z.x, ub)));
      if (k == 0) {  // the shift's own mode
        A.x += N * bits_double(fa);
        B.x += N * bits_double(fb);
      }
      if (ea == kNanExp) A = make_double2(bits_double(kNan), bits_double(kNan));
      if (eb == kNanExp) B = make_double2(bits_double(kNan), bits_double(kNan));
      Fa[k] = A;
      Fa[HX + k] = B;
    }
    __syncwarp();  // the modes are read before the next tile's values replace them
  }
}

// Complex lines in place: line l starts at base(l), its points `stride` apart;
// 16 neighbouring lines are contiguous (but for the rows' ends along y).
// per: lines of one plane (along y: nx/2+1 per z; along z: all).
template <int N>
__global__ void __launch_bounds__(Geo<N>::THREADS, Geo<N>::MINB) fxr_lines(double2* F, int64_t nlines, int per,
                                                                           int64_t plane, int64_t stride,
                                                                           const Tw* tw) {
  using G = Geo<N>;
  constexpr int P = G::P, Q = G::Q, W = P / 2, GR = Q / P;
  extern __shared__ __align__(16) unsigned char smraw[];
  Tw* t1 = reinterpret_cast<Tw*>(smraw);
  Cx64* scratch = reinterpret_cast<Cx64*>(t1 + N);
  __shared__ int emx[W][kLines];
  __shared__ u64 ors[W][kLines], sums[W][kLines];
  const int tid = threadIdx.x, warp = tid >> 5, t = tid / kLines, li = tid % kLines;
  Cx64* sl = scratch + li * G::LSTRIDE;
  load_twiddles<N>(tw, t1, tid);
  __syncthreads();
  auto imax = [](int x, int y) { return max(x, y); };
  auto oor = [](u64 x, u64 y) { return x | y; };
  auto add = [](u64 x, u64 y) { return x + y; };
  const int64_t ntile = nlines / kLines;
  for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int64_t l = tile * kLines + li;
    double2* f = F + (l / per) * plane + l % per;
    int e = 1;
#pragma unroll 8
    for (int q = 0; q < Q; ++q) {
      const double2 v = f[(t + P * q) * stride];
      const u64 bx = double_bits(v.x), by = double_bits(v.y);
      e = max(e, max(exp_of(bx), exp_of(by)));
      sl[q * G::S + t] = Cx64{(i64)bx, (i64)by};
    }
    e = line_reduce<1, P>(e, imax, emx, li, warp);
    __syncthreads();
    e = line_collect<1, P>(e, imax, emx, li);
    u64 o = 0, s = 2 * Q;
#pragma unroll 4
    for (int q = 0; q < Q; ++q) {
      Cx64 z = sl[q * G::S + t];
      z.x = from_bits((u64)z.x, e);
      z.y = from_bits((u64)z.y, e);
      sl[q * G::S + t] = z;
      const u64 mx = (u64)(z.x ^ (z.x >> 63)), my = (u64)(z.y ^ (z.y >> 63));
      o |= mx | my;
      s += (mx >> 9) + (my >> 9);
    }
    o = line_reduce<1, P>(o, oor, ors, li, warp);
    s = line_reduce<1, P>(s, add, sums, li, warp);
    __syncthreads();
    o = line_collect<1, P>(o, oor, ors, li);
    s = line_collect<1, P>(s, add, sums, li);
    const LineBits b = line_bits<2 * N, Split<N>::LOG + 1>(o, s);
    i64 re[Q], im[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const Cx64 z = sl[q * G::S + t];
      re[q] = scale_line(z.x, b);
      im[q] = scale_line(z.y, b);
    }
    phase1<N>(re, im, t, sl, t1);
    __syncthreads();
    phase2_forward<N>(t, sl);
    const int u = emax_unit(e, b);
    for (int g = 0; g < GR; ++g) {  // the thread's own rows
      const int kq = t + g * P;
#pragma unroll 4
      for (int kp = 0; kp < P; ++kp) {
        const Cx64 z = sl[kq * G::S + kp];
        double2 v = make_double2(bits_double(to_bits_exp(z.x, u)), bits_double(to_bits_exp(z.y, u)));
        if (e == kNanExp) v = make_double2(bits_double(kNan), bits_double(kNan));
        f[(kq + Q * kp) * stride] = v;
      }
    }
    __syncthreads();  // the rows are read before the next tile's values replace them
  }
}

template <int N>
int fxr_rows_go(const RowIn& in, bool f32, double2* F, int64_t nlines, const Tw* tw, int nsm, cudaStream_t s) {
  using G = Geo<N>;
  const int smem = (N + kLines * G::LSTRIDE) * 16;
  if (nlines % kLines) return set_error(LAT_ERR_STATE, "fixed-point transform: partial tile");
  auto k64 = fxr_rows<N, false>;
  auto k32 = fxr_rows<N, true>;
  cudaError_t e = cudaFuncSetAttribute(f32 ? k32 : k64, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, "fixed-point transform smem attribute");
  const int grid = (int)std::min<int64_t>(nlines / kLines, (int64_t)nsm * G::MINB);
  if (f32) k32<<<grid, G::THREADS, smem, s>>>(in, F, nlines, tw);
  else k64<<<grid, G::THREADS, smem, s>>>(in, F, nlines, tw);
  if (g_launch_counter) ++*g_launch_counter;
  e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, "fixed-point transform launch");
}
template <int N>
int fxr_lines_go(double2* F, int64_t nlines, int per, int64_t plane, int64_t stride, const Tw* tw, int nsm,
                 cudaStream_t s) {
  using G = Geo<N>;
  const int smem = (N + kLines * G::LSTRIDE) * 16;
  if (nlines % kLines) return set_error(LAT_ERR_STATE, "fixed-point transform: partial tile");
  auto k = fxr_lines<N>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, "fixed-point transform smem attribute");
  const int grid = (int)std::min<int64_t>(nlines / kLines, (int64_t)nsm * G::MINB);
  k<<<grid, G::THREADS, smem, s>>>(F, nlines, per, plane, stride, tw);
  if (g_launch_counter) ++*g_launch_counter;
  e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, "fixed-point transform launch");
}

}  // namespace fx
}  // namespace lat
