// k_bin.cu -- shell binning of half spectra: power, cross and TT-projected
// gravitational-wave spectra.
//
// spectrum_3d / crossspec_3d (Pseudospec/openmp_dev/analysis_spec.f90:59-102,
// 145-178; two-bin weights c0 = (1 - (l - p)^2)^2 into shell l = floor(p) and
// c1 into l + 1, p = |n|) and spectrum_bin (Discrete/Bubble-Collisions/
// analysis.f90:193-223; shell l, integer counts).  The reference loops over the
// full x range with folded indices, i.e. Hermitian weight 2 on interior kx
// planes.
//
// The sums are FP64, and GB300 runs 2 FP64 operations per clock and SM, so the
// design spends as few as it can.  The rows (+-y, +-z) share |n| at every x: a
// warp adds their (up to four) values first and weights the sum once; weights
// come from a table over |n|^2 and the weight sums W, which hold no data, from
// the lattice's plan.  Along a row the shells ascend, so the lanes of one shell
// are neighbours: a segmented shuffle sum leaves one addition per shell to the
// warp's own bins in shared memory, with no atomics and in a fixed order.
// Two-bin power spectrum of a 256^3 lattice: 0.12 ms; 0.62 with one FP64 square
// root, eight weight operations and four shared-memory atomics a mode.
#include <algorithm>
#include <string>
#include <vector>

#include "bin.hpp"

namespace lat {

namespace {

enum { BIN_POWER = 0, BIN_COUNT = 1, BIN_CROSS = 2, BIN_GW = 3 };
template <int KIND> struct Sums { static constexpr int NS = KIND == BIN_POWER ? 2 : (KIND == BIN_CROSS ? 4 : 1); };

// sum_ij |h^TT_ij|^2 of one mode: with e1, e2 normal to k,
// 1/2 |e1 h e1 - e2 h e2|^2 + 2 |e1 h e2|^2, written out for
// e1 = (-ky, kx, 0)/rho, e2 = (-kx kz, -ky kz, rho^2)/(rho k), rho^2 = kx^2 + ky^2
// (k along z: e1 = x, e2 = y).  The projector P pi P - P tr(P pi)/2 of
// grav-waves/gw-projectors.f90:13-26 without its 3 x 3 products.
template <typename C>
__device__ __forceinline__ double tt_power(const C (&h)[6], double kx, double ky, double kz) {
  const double x2 = kx * kx, y2 = ky * ky, z2 = kz * kz, rho2 = x2 + y2, k2 = rho2 + z2;
  if (!(k2 > 0.0)) return 0.0;
  double re[6], im[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    re[i] = widen(h[i].x);
    im[i] = widen(h[i].y);
  }
  if (rho2 == 0.0) {
    const double dr = re[0] - re[1], di = im[0] - im[1];
    return 0.5 * (dr * dr + di * di) + 2.0 * (re[3] * re[3] + im[3] * im[3]);
  }
  // (e1 h e1 - e2 h e2) rho^2 k^2 and (e1 h e2) rho^2 k
  const double xy = kx * ky, a11 = y2 * k2 - x2 * z2, a22 = x2 * k2 - y2 * z2, a33 = -rho2 * rho2;
  const double a12 = -2.0 * xy * (k2 + z2), rz = 2.0 * rho2 * kz, a13 = rz * kx, a23 = rz * ky;
  const double c1 = xy * kz, c2 = kz * (y2 - x2), c3 = rho2 * kx, c4 = rho2 * ky;
  const double dr = a11 * re[0] + a22 * re[1] + a33 * re[2] + a12 * re[3] + a13 * re[4] + a23 * re[5];
  const double di = a11 * im[0] + a22 * im[1] + a33 * im[2] + a12 * im[3] + a13 * im[4] + a23 * im[5];
  const double er = c1 * (re[0] - re[1]) + c2 * re[3] + c3 * re[5] - c4 * re[4];
  const double ei = c1 * (im[0] - im[1]) + c2 * im[3] + c3 * im[5] - c4 * im[4];
  const double d = rho2 * k2;
  return (0.5 * (dr * dr + di * di) + 2.0 * k2 * (er * er + ei * ei)) / (d * d);
}

template <int KIND, typename C>
__global__ void __launch_bounds__(256) bin_kernel(BinArgs a) {
  constexpr int NS = Sums<KIND>::NS;
  constexpr unsigned int full = 0xffffffffu;
  extern __shared__ double bins[];  // [warps][NS][nb]
  __shared__ int am_last;
  const int nb = a.nbins, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* mine = bins + (size_t)warp * NS * nb;
  for (int i = lane; i < NS * nb; i += 32) mine[i] = 0.0;
  __syncwarp();
  const int hx = a.nx / 2 + 1, hy = a.ny / 2 + 1, hz = a.nz / 2 + 1;
  const C* F1 = static_cast<const C*>(a.F[0]);
  const C* F2 = static_cast<const C*>(a.F[1]);
  const int nrow = hy * hz, xend = min(hx, nb);
  for (int row = blockIdx.x * nw + warp; row < nrow; row += gridDim.x * nw) {
    const int jj = row % hy, kk = row / hy;
    if (jj >= nb || kk >= nb) continue;  // beyond the last shell, as the x from nb on: |n|^2 stays below 3 nb^2
    const int r2 = jj * jj + kk * kk;
    const int my = (jj == 0 || 2 * jj == a.ny) ? 1 : 2, mz = (kk == 0 || 2 * kk == a.nz) ? 1 : 2;
    size_t at[4];  // the rows (+-y, +-z)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int y = my == 2 && (r & 1) ? a.ny - jj : jj, z = (my == 2 ? r >> 1 : r) ? a.nz - kk : kk;
      at[r] = ((size_t)z * a.ny + y) * hx;
    }
    for (int x0 = 0; x0 < xend; x0 += 32) {
      const int x = x0 + lane;
      const bool on = x < xend;
      const int m2 = r2 + x * x, l = on ? isqrt_exact(m2) : 0x40000000 + lane;
      double v = 0.0, vi = 0.0;
      if constexpr (KIND == BIN_GW) {
        if (on && l < nb) {
          for (int r = 0; r < my * mz; ++r) {
            C h[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) h[i] = static_cast<const C*>(a.F[i])[at[r] + x];
            const int y = (r & 1) && my == 2 ? a.ny - jj : jj, z = r >= my ? a.nz - kk : kk;
            v += tt_power(h, __ldg(a.sins + x), __ldg(a.sins + hx + y), __ldg(a.sins + hx + a.ny + z));
          }
        }
      } else {
        // the mirrored rows' values in flight together
        C f[4], g[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          f[r] = C{0, 0};
          g[r] = C{0, 0};
          if (on && r < my * mz) {
            f[r] = F1[at[r] + x];
            if constexpr (KIND == BIN_CROSS) g[r] = F2[at[r] + x];
          }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (r >= my * mz) break;
          const double fr = widen(f[r].x), fi = widen(f[r].y);
          if constexpr (KIND == BIN_CROSS) {
            const double gr = widen(g[r].x), gi = widen(g[r].y);
            v = fma(fi, gi, fma(fr, gr, v));     // Re(F1 conj F2)
            vi = fma(-fr, gi, fma(fi, gr, vi));  // Im(F1 conj F2)
          } else {
            v = fma(fi, fi, fma(fr, fr, v));
          }
        }
      }
      if (x != 0 && 2 * x != a.nx) {
        v += v;
        vi += vi;
      }
      double s[NS];
      if constexpr (KIND == BIN_POWER || KIND == BIN_CROSS) {
        const double2 c = on && l < nb ? __ldg(a.wtab + m2) : make_double2(0.0, 0.0);  // m2 < nb^2
        s[0] = c.x * v;
        s[1] = c.y * v;
        if constexpr (KIND == BIN_CROSS) {
          s[2] = c.x * vi;
          s[3] = c.y * vi;
        }
      } else {
        s[0] = v;
      }
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_down_sync(full, l, d);
        const bool same = lane + d < 32 && o == l;
        if (!__any_sync(full, same)) break;
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          const double w = __shfl_down_sync(full, s[i], d);
          if (same) s[i] += w;
        }
      }
      const int before = __shfl_up_sync(full, l, 1);
      if ((lane == 0 || before != l) && l < nb) {
#pragma unroll
        for (int i = 0; i < NS; ++i) mine[i * nb + l] += s[i];
      }
      __syncwarp();
    }
  }
  __syncthreads();
  // the block's warps, then the grid's blocks, in order
  for (int i = threadIdx.x; i < NS * nb; i += blockDim.x) {
    double s = bins[i];
    for (int w = 1; w < nw; ++w) s += bins[(size_t)w * NS * nb + i];
    a.partials[(size_t)blockIdx.x * NS * nb + i] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) am_last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  for (int i = threadIdx.x; i < NS * nb; i += blockDim.x) {
    double s = 0.0;
#pragma unroll 8
    for (int b = 0; b < (int)gridDim.x; ++b) s += __ldcg(a.partials + (size_t)b * NS * nb + i);
    a.out[i] = s;
  }
  if (threadIdx.x == 0) *a.counter = 0u;
}

// ------------------------------------------------------------- the plan
// weights of the two bins of a mode at |n|^2 = m2; the correctly rounded FP64
// square root and uncontracted arithmetic give the host's bits
__global__ void bin_weight_kernel(double2* wtab, int n) {
  for (int m2 = blockIdx.x * blockDim.x + threadIdx.x; m2 < n; m2 += gridDim.x * blockDim.x) {
    const int l = isqrt_exact(m2);
    const double p = sqrt((double)m2);
    const double d0 = __dsub_rn((double)l, p), d1 = __dsub_rn((double)(l + 1), p);
    const double e0 = __dsub_rn(1.0, __dmul_rn(d0, d0)), e1 = __dsub_rn(1.0, __dmul_rn(d1, d1));
    wtab[m2] = make_double2(__dmul_rn(e0, e0), __dmul_rn(e1, e1));
  }
}
// modes of the full spectrum at every |n|^2 below n
__global__ void bin_count_kernel(int* cnt, int n, int nx, int ny, int nz) {
  const int hx = nx / 2 + 1, hy = ny / 2 + 1, hz = nz / 2 + 1;
  const long long tot = (long long)hx * hy * hz;
  auto mult = [](int i, int n) { return i == 0 || 2 * i == n ? 1 : 2; };
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(t % hx), y = (int)(t / hx % hy), z = (int)(t / hx / hy);
    const long long m2 = (long long)x * x + (long long)y * y + (long long)z * z;
    if (m2 < n) atomicAdd(cnt + m2, mult(x, nx) * mult(y, ny) * mult(z, nz));
  }
}
// W[l]: two-bin weight sums, W[nb + l]: counts; one warp per shell
__global__ void bin_sum_kernel(const int* cnt, const double2* wtab, int n, int nb, double* W) {
  const int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (l >= nb) return;
  double w = 0.0, c = 0.0;
  const int end = min((l + 1) * (l + 1), n);
  for (int m2 = (l ? (l - 1) * (l - 1) : 0) + lane; m2 < end; m2 += 32) {
    const double k = (double)cnt[m2];
    const double2 t = wtab[m2];
    if (m2 >= l * l) {
      w += k * t.x;
      c += k;
    } else {
      w += k * t.y;
    }
  }
  w = warp_sum(w);
  c = warp_sum(c);
  if (lane == 0) {
    W[l] = w;
    W[nb + l] = c;
  }
}
// sin(2 pi i / n), the lattice momentum of the central difference times dx
__global__ void bin_sin_kernel(double* s, int nx, int ny, int nz) {
  const double twopi = 6.283185307179586476925286766559;
  const int hx = nx / 2 + 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < hx + ny + nz; i += gridDim.x * blockDim.x)
    s[i] = i < hx ? sin(twopi * i / nx) : (i < hx + ny ? sin(twopi * (i - hx) / ny) : sin(twopi * (i - hx - ny) / nz));
}

template <int KIND>
int bin_go(BinArgs a, int precision, int nsm, cudaStream_t s) {
  const size_t per = (size_t)Sums<KIND>::NS * a.nbins * sizeof(double);  // one warp's bins
  constexpr size_t most = 96 * 1024;
  int warps = 8;
  while (warps > 1 && warps * per > most) warps /= 2;
  const size_t smem = warps * per;
  auto k64 = bin_kernel<KIND, double2>;
  auto k32 = bin_kernel<KIND, float2>;
  // the limit belongs to the kernel, not to the call: always the largest size,
  // which another thread's call may be about to launch with (and always, as the
  // static shared memory counts towards the default 48 KB too)
  const cudaError_t es = cudaFuncSetAttribute(precision == LAT_FP64 ? k64 : k32,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (es != cudaSuccess) return cuda_fail(es, "binning smem attribute");
  const int rows = (a.ny / 2 + 1) * (a.nz / 2 + 1);
  const int grid = std::min(2 * nsm, (rows + warps - 1) / warps);
  if (precision == LAT_FP64) k64<<<grid, 32 * warps, smem, s>>>(a);
  else k32<<<grid, 32 * warps, smem, s>>>(a);
  if (g_launch_counter) ++*g_launch_counter;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, "binning launch");
}

}  // namespace

int BinPlan::make(int nx_, int ny_, int nz_, int nsm_, cudaStream_t s) {
  if (wtab) return LAT_OK;
  nx = nx_;
  ny = ny_;
  nz = nz_;
  nsm = nsm_;
  // one allocation: weights, sines, output, counter, and the partial sums,
  // whose space first holds the counts and the weight sums
  const int n = (int)bin_table_size(nx, ny, nz);
  const size_t ns = (size_t)(nx / 2 + 1) + ny + nz, no = (size_t)4 * kMaxBins;
  const size_t np = std::max<size_t>(no * 2 * nsm, 2 * kMaxBins + ((size_t)n + 1) / 2);
  double* mem = nullptr;
  cudaError_t e = cudaMalloc(&mem, sizeof(double) * (2 * (size_t)n + ns + no + 8 + np));
  if (e != cudaSuccess) return set_error(LAT_ERR_ALLOC, std::string("spectrum tables: ") + cudaGetErrorString(e));
  wtab = reinterpret_cast<double2*>(mem);
  sins = mem + 2 * (size_t)n;
  out = sins + ns;
  counter = reinterpret_cast<unsigned int*>(out + no);
  partials = out + no + 8;
  double* W = partials;
  int* cnt = reinterpret_cast<int*>(partials + 2 * kMaxBins);
  std::vector<double> w(2 * kMaxBins);
  e = cudaMemsetAsync(counter, 0, 64, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, sizeof(int) * n, s);
  if (e == cudaSuccess) {
    const long long oct = (long long)(nx / 2 + 1) * (ny / 2 + 1) * (nz / 2 + 1);
    bin_weight_kernel<<<std::min((n + 255) / 256, 4 * nsm), 256, 0, s>>>(wtab, n);
    bin_sin_kernel<<<8, 128, 0, s>>>(sins, nx, ny, nz);
    bin_count_kernel<<<(int)std::min<long long>((oct + 255) / 256, 8 * nsm), 256, 0, s>>>(cnt, n, nx, ny, nz);
    bin_sum_kernel<<<kMaxBins / 8, 256, 0, s>>>(cnt, wtab, n, kMaxBins, W);
    if (g_launch_counter) *g_launch_counter += 4;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(w.data(), W, sizeof(double) * 2 * kMaxBins, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    free();
    return cuda_fail(e, "spectrum tables");
  }
  Ww.assign(w.begin(), w.begin() + kMaxBins);
  Wc.assign(w.begin() + kMaxBins, w.end());
  return LAT_OK;
}

void BinPlan::free() {
  if (wtab) cudaFree(wtab);
  wtab = nullptr;
}

int BinPlan::sums(int kind, const void* const* F, int nf, int precision, int nbins, std::vector<double>& o,
                  cudaStream_t s) {
  BinArgs a{};
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.nbins = nbins;
  for (int i = 0; i < nf; ++i) a.F[i] = F[i];
  a.wtab = wtab;
  a.sins = sins;
  a.partials = partials;
  a.out = out;
  a.counter = counter;
  int st, ns;
  switch (kind) {
    case BIN_POWER: st = bin_go<BIN_POWER>(a, precision, nsm, s); ns = 2; break;
    case BIN_COUNT: st = bin_go<BIN_COUNT>(a, precision, nsm, s); ns = 1; break;
    case BIN_CROSS: st = bin_go<BIN_CROSS>(a, precision, nsm, s); ns = 4; break;
    default: st = bin_go<BIN_GW>(a, precision, nsm, s); ns = 1;
  }
  if (st != LAT_OK) return st;
  o.resize((size_t)ns * nbins);
  cudaError_t e = cudaMemcpyAsync(o.data(), out, sizeof(double) * o.size(), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, "spectrum read-back");
}

int BinPlan::power(const void* F, int mode, int precision, int nbins, double* S, double* W, cudaStream_t s) {
  std::vector<double> o;
  const bool two = mode == LAT_SPEC_WEIGHTED;
  const int st = sums(two ? BIN_POWER : BIN_COUNT, &F, 1, precision, nbins, o, s);
  if (st != LAT_OK) return st;
  for (int l = 0; l < nbins; ++l) {
    const double v = two ? o[l] + (l ? o[nbins + l - 1] : 0.0) : o[l];
    W[l] = two ? Ww[l] : Wc[l];
    S[l] = W[l] != 0.0 ? v / W[l] : v;
  }
  return LAT_OK;
}

int BinPlan::cross(const void* F1, const void* F2, int precision, int nbins, double* S_re, double* S_im,
                   cudaStream_t s) {
  std::vector<double> o;
  const void* F[2] = {F1, F2};
  const int st = sums(BIN_CROSS, F, 2, precision, nbins, o, s);
  if (st != LAT_OK) return st;
  for (int l = 0; l < nbins; ++l) {
    const double re = o[l] + (l ? o[nbins + l - 1] : 0.0);
    const double im = o[2 * nbins + l] + (l ? o[3 * nbins + l - 1] : 0.0);
    S_re[l] = Ww[l] != 0.0 ? re / Ww[l] : re;
    S_im[l] = Ww[l] != 0.0 ? im / Ww[l] : im;
  }
  return LAT_OK;
}

int BinPlan::gw(const void* const* F, int precision, int nbins, double* S, double* W, cudaStream_t s) {
  std::vector<double> o;
  const int st = sums(BIN_GW, F, 6, precision, nbins, o, s);
  if (st != LAT_OK) return st;
  for (int l = 0; l < nbins; ++l) {
    W[l] = Wc[l];
    S[l] = W[l] != 0.0 ? o[l] / W[l] : o[l];
  }
  return LAT_OK;
}

}  // namespace lat
