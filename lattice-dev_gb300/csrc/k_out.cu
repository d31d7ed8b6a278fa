// k_out.cu -- layout conversion and initial conditions.
#include "engine.hpp"

namespace lat {

namespace {

// ------------------------------------------------------------ layouts
// Fortran fld(nfld, i, j, k) (field fastest) <-> device [field][z][y][x].
template <typename R, bool KAHAN>
// fs: element stride between fields of the SoA side (N, or the plane count
// of a z-slab's storage times the plane size when N covers its interior)
__global__ void aos2soa_kernel(const double* __restrict__ aos, int nf, int64_t N, int64_t fs, R* hi, R* c) {
  const int64_t tot = N * nf;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = t / nf;
    const int f = (int)(t - s * nf);
    const double v = aos[t];
    const R h = (R)v;
    hi[f * fs + s] = h;
    if (KAHAN && c) c[f * fs + s] = (R)((double)h - v);
  }
}
template <typename R, bool KAHAN>
__global__ void soa2aos_kernel(const R* hi, const R* c, int nf, int64_t N, int64_t fs, double* __restrict__ aos) {
  const int64_t tot = N * nf;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = t / nf;
    const int f = (int)(t - s * nf);
    double v = (double)hi[f * fs + s];
    if (KAHAN && c) v -= (double)c[f * fs + s];
    aos[t] = v;
  }
}
template <typename R, bool KAHAN>
__global__ void to64_kernel(const R* hi, const R* c, int64_t n, double* out) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    double v = (double)hi[t];
    if (KAHAN && c) v -= (double)c[t];
    out[t] = v;
  }
}
template <typename R, bool KAHAN>
__global__ void from64_kernel(const double* in, int64_t n, R* hi, R* c) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const double v = in[t];
    const R h = (R)v;
    hi[t] = h;
    if (KAHAN && c) c[t] = (R)((double)h - v);
  }
}

inline int grid_for(int64_t n) {
  int64_t g = (n + 255) / 256;
  return (int)(g > 4096 ? 4096 : (g < 1 ? 1 : g));
}
inline int done(const char* what) {
  if (g_launch_counter) ++*g_launch_counter;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, what);
}

// -------------------------------------------------- initial conditions
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double u01(uint64_t r) { return ((double)(r >> 11) + 1.0) * (1.0 / 9007199254740992.0); }
__device__ __forceinline__ double2 mode_gauss(uint64_t seed, int field, int64_t mode) {
  const uint64_t key = mix64(mix64(mix64(seed) ^ (uint64_t)field) ^ (uint64_t)mode);
  const double u1 = u01(mix64(key ^ 1ULL)), u2 = u01(mix64(key ^ 2ULL));
  const double r = sqrt(-2.0 * log(u1));
  const double th = 6.2831853071795864769252867665590 * u2;
  return make_double2(r * cos(th), r * sin(th));
}

// Same draw as the oracle's orc_init_vacuum: Hermitian partners inside the
// kx = 0 and kx = nx/2 planes share one draw (the lower mode index draws).
__global__ void vacuum_kernel(VacArgs a) {
  const int hx = a.nx / 2 + 1;
  const int64_t M = (int64_t)hx * a.ny * a.nz;
  for (int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(m % hx);
    const int64_t r = m / hx;
    const int y = (int)(r % a.ny), z = (int)(r / a.ny);
    const int jj = fold_idx(y, a.ny), kk = fold_idx(z, a.nz);
    const double k2 = (double)x * x * a.dkx * a.dkx + (double)jj * jj * a.dky * a.dky + (double)kk * kk * a.dkz * a.dkz;
    double2 F = make_double2(0, 0), P = make_double2(0, 0);
    if (k2 > 0.0 && sqrt(k2) <= a.kcut) {
      const double w = sqrt(k2 + a.m2);
      const double sig = sqrt(a.sig_pref / w);
      const bool selfplane = (x == 0) || (2 * x == a.nx);
      const int64_t mp = ((int64_t)((a.nz - z) % a.nz) * a.ny + (a.ny - y) % a.ny) * hx + x;
      const double h = 0.70710678118654752440084436210485;
      // pi_k = -i w F_k for the drawing member of a pair (a wave travelling along
      // +k); the Hermitian partner carries +i w F, a self-conjugate mode none.
      if (selfplane && mp == m) {
        double2 g = mode_gauss(a.seed, a.field, m);
        F = make_double2(sig * g.x, 0.0);
      } else if (selfplane && mp < m) {
        double2 g = mode_gauss(a.seed, a.field, mp);
        F = make_double2(sig * g.x * h, -(sig * g.y * h));
        P = make_double2(-w * F.y, w * F.x);  // +i w F
      } else {
        double2 g = mode_gauss(a.seed, a.field, m);
        F = make_double2(sig * g.x * h, sig * g.y * h);
        P = make_double2(w * F.y, -w * F.x);  // -i w F
      }
    }
    a.Fphi[m] = F;
    a.Fpi[m] = P;
  }
}

// ------------------------------------------- the reference's sample() IC
// (Pseudospec/openmp_dev/evolve_spectral.f90:421-506).  The DST-II of the
// oversampled radial profile, Y_k = 2 sum_j X_j sin(pi (2j+1)(k+1) / (2 nos)),
// is the imaginary part of one complex FFT of length 4 nos of the odd
// embedding z[2j+1] = X_j, z[4 nos - 2j - 1] = -X_j: Y_k = -Im Z_{k+1}.
__global__ void sample_dst_in_kernel(double2* z, int nos, double dkos, double m2, double gamma, double kcut) {
  const int64_t L4 = 4LL * nos;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < L4; t += (int64_t)gridDim.x * blockDim.x) {
    double v = 0.0;
    if (t & 1) {
      const bool lower = t < 2LL * nos;
      const int64_t j = lower ? (t - 1) / 2 : (L4 - t - 1) / 2;
      const double kk = (j + 0.5) * dkos;
      const double x = kk * pow(kk * kk + m2, gamma) * exp(-(kk / kcut) * (kk / kcut));
      v = lower ? x : -x;
    }
    z[t] = make_double2(v, 0.0);
  }
}

// ker[k] = norm Y_k / (k + 1): the 1-based profile ker(k + 1)
__global__ void sample_dst_out_kernel(const double2* Z, int nos, double norm, double* ker) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nos; t += gridDim.x * blockDim.x)
    ker[t] = norm * (-Z[t + 1].y) / (t + 1);
}

// the profile interpolated at |(i, j, k) - nn| os (1-based indices, nn = n/2 + 1)
__global__ void sample_kernel3d(const double* ker, int n, double* f) {
  const int64_t N = (int64_t)n * n * n;
  const int nn = n / 2 + 1, os = 16;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(t % n), y = (int)((t / n) % n), z = (int)(t / ((int64_t)n * n));
    const double di = x + 1 - nn, dj = y + 1 - nn, dz = z + 1 - nn;
    const double kk = sqrt(di * di + dj * dj + dz * dz) * os;
    const int l = (int)floor(kk);
    f[t] = l > 0 ? ker[l - 1] + (kk - l) * (ker[l] - ker[l - 1]) : (4.0 * ker[0] - ker[1]) / 3.0;
  }
}

// every half-spectrum mode times the Box-Muller noise of its counter-based draw
__global__ void sample_noise_kernel(double2* F, int64_t M, uint64_t seed, int stream) {
  for (int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (int64_t)gridDim.x * blockDim.x) {
    const double2 g = mode_gauss(seed, stream, m), v = F[m];
    F[m] = make_double2(v.x * g.x - v.y * g.y, v.x * g.y + v.y * g.x);
  }
}

// the kx = 0 and kx = n/2 planes projected onto their Hermitian part
__global__ void sample_hermitize_kernel(double2* F, int n) {
  const int hx = n / 2 + 1;
  const int64_t P = 2LL * n * n;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < P; t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (t < (int64_t)n * n) ? 0 : n / 2;
    const int64_t r = t % ((int64_t)n * n);
    const int y = (int)(r % n), z = (int)(r / n);
    const int64_t m = ((int64_t)z * n + y) * hx + x;
    const int64_t mp = ((int64_t)((n - z) % n) * n + (n - y) % n) * hx + x;
    if (mp < m) continue;
    const double2 a = F[m], b = F[mp];
    const double2 h = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    F[m] = h;
    F[mp] = make_double2(h.x, -h.y);
  }
}

// STENCIL(c,LAPLACE) with pre-scaled coefficients lc = c/(cc dx^2), FP64.
__global__ void fd_lap64_kernel(const double* g, double* out, int nx, int ny, int nz, double l0, double l1, double l2,
                                double l3) {
  const int64_t N = (int64_t)nx * ny * nz;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(t % nx), y = (int)((t / nx) % ny), z = (int)(t / ((int64_t)nx * ny));
    double r1 = 0, r2 = 0, r3 = 0;
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
          const int rank = (dx != 0) + (dy != 0) + (dz != 0);
          if (rank == 0) continue;
          const int xx = x + dx < 0 ? x + dx + nx : (x + dx >= nx ? x + dx - nx : x + dx);
          const int yy = y + dy < 0 ? y + dy + ny : (y + dy >= ny ? y + dy - ny : y + dy);
          const int zz = z + dz < 0 ? z + dz + nz : (z + dz >= nz ? z + dz - nz : z + dz);
          const double v = g[((int64_t)zz * ny + yy) * nx + xx];
          if (rank == 1) r1 += v; else if (rank == 2) r2 += v; else r3 += v;
        }
    out[t] = l0 * g[t] + l1 * r1 + l2 * r2 + l3 * r3;
  }
}

__global__ void add_scale_kernel(double* f, int64_t n, double scale, double offset) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    f[t] = offset + f[t] * scale;
}

__global__ void bubbles_kernel(double* phi, int nx, int ny, int nz, double dx, int nbub, const double* cen,
                               double R, double w) {
  const int64_t N = (int64_t)nx * ny * nz;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(t % nx), y = (int)((t / nx) % ny), z = (int)(t / ((int64_t)nx * ny));
    double v = -1.0;
    for (int b = 0; b < nbub; ++b) {
      const double rx = x * dx - cen[3 * b], ry = y * dx - cen[3 * b + 1], rz = z * dx - cen[3 * b + 2];
      const double rr = sqrt(rx * rx + ry * ry + rz * rz);
      v += 1.0 - tanh((rr - R) / w);
    }
    phi[t] = v;
  }
}

// Boosted-wall bubbles of Discrete/Bubble-Collisions/ic_bubble.f90:45-77 with
// the profile and time derivative of init_cond.f90:192-234: centres are
// 1-based site indices, distances are not wrapped, bubbles superpose, and
// phi_false is added at the end.
__global__ void bubbles_boost_kernel(double* phi, double* pi, int nx, int ny, int nz, double dx, int nbub,
                                     const int* cen, double r0, double t0, double pf, double pt) {
  const int64_t N = (int64_t)nx * ny * nz;
  const double step = (pf - pt) / 2.0, ave = (-pf + pt) / 2.0, rt2 = 1.4142135623730951;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(t % nx), y = (int)((t / nx) % ny), z = (int)(t / ((int64_t)nx * ny));
    double f = 0.0, d = 0.0;
    for (int b = 0; b < nbub; ++b) {
      const int ii = x + 1 - cen[3 * b], jj = y + 1 - cen[3 * b + 1], kk = z + 1 - cen[3 * b + 2];
      const double rad = sqrt((double)(ii * ii + jj * jj + kk * kk) * dx * dx);
      if (rad * rad > t0 * t0) {
        const double s1 = sqrt(rad * rad - t0 * t0), s = s1 - r0;
        const double ch = cosh(s / rt2);
        f += step * tanh(s / rt2) + ave;
        d += -step * t0 / s1 / rt2 / (ch * ch);
      } else {
        f += pt - pf;
      }
    }
    phi[t] = f + pf;
    pi[t] = d;
  }
}

}  // namespace

int launch_bubbles_boosted(double* phi, double* pi, int nx, int ny, int nz, double dx, int nbub, const int* cen,
                           double r0, double t0, double pf, double pt, cudaStream_t s) {
  bubbles_boost_kernel<<<grid_for((int64_t)nx * ny * nz), 256, 0, s>>>(phi, pi, nx, ny, nz, dx, nbub, cen, r0, t0,
                                                                       pf, pt);
  return done("boosted bubbles");
}

int launch_aos2soa(const double* aos, int nf, int64_t N, int precision, void* hi, void* c, cudaStream_t s,
                   int64_t fstride) {
  const int64_t fs = fstride > 0 ? fstride : N;
  if (precision == LAT_FP64)
    aos2soa_kernel<double, false><<<grid_for(N * nf), 256, 0, s>>>(aos, nf, N, fs, (double*)hi, nullptr);
  else aos2soa_kernel<float, true><<<grid_for(N * nf), 256, 0, s>>>(aos, nf, N, fs, (float*)hi, (float*)c);
  return done("aos2soa");
}
int launch_soa2aos(const void* hi, const void* c, int nf, int64_t N, int precision, double* aos, cudaStream_t s,
                   int64_t fstride) {
  const int64_t fs = fstride > 0 ? fstride : N;
  if (precision == LAT_FP64)
    soa2aos_kernel<double, false><<<grid_for(N * nf), 256, 0, s>>>((const double*)hi, nullptr, nf, N, fs, aos);
  else
    soa2aos_kernel<float, true><<<grid_for(N * nf), 256, 0, s>>>((const float*)hi, (const float*)c, nf, N, fs, aos);
  return done("soa2aos");
}
// Every ds-th site of one field array as FP64 (phi_hi - c for FP32), in the
// lattice order (x fastest): the data of output_cube
// (Discrete/Bubble-Collisions/outputfile.f90:942-1016).
template <typename R, bool KAHAN>
__global__ void cube_kernel(const R* __restrict__ hi, const R* __restrict__ c, int nx, int ny, int nz, int ds,
                            double* __restrict__ out) {
  const int mx = nx / ds, my = ny / ds, mz = nz / ds;
  const int64_t M = (int64_t)mx * my * mz;
  for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < M; o += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(o % mx), j = (int)((o / mx) % my), k = (int)(o / ((int64_t)mx * my));
    const int64_t s = ((int64_t)k * ds * ny + (int64_t)j * ds) * nx + (int64_t)i * ds;
    out[o] = KAHAN ? (double)hi[s] - (double)c[s] : (double)hi[s];
  }
}

int launch_cube(const void* hi, const void* c, int nx, int ny, int nz, int ds, int precision, double* out,
                cudaStream_t s) {
  const int64_t M = (int64_t)(nx / ds) * (ny / ds) * (nz / ds);
  if (precision == LAT_FP64)
    cube_kernel<double, false><<<grid_for(M), 256, 0, s>>>((const double*)hi, nullptr, nx, ny, nz, ds, out);
  else if (c)
    cube_kernel<float, true><<<grid_for(M), 256, 0, s>>>((const float*)hi, (const float*)c, nx, ny, nz, ds, out);
  else
    cube_kernel<float, false><<<grid_for(M), 256, 0, s>>>((const float*)hi, nullptr, nx, ny, nz, ds, out);
  return done("cube");
}

int launch_to_fp64(const void* hi, const void* c, int64_t n, int precision, double* out, cudaStream_t s) {
  if (precision == LAT_FP64) to64_kernel<double, false><<<grid_for(n), 256, 0, s>>>((const double*)hi, nullptr, n, out);
  else to64_kernel<float, true><<<grid_for(n), 256, 0, s>>>((const float*)hi, (const float*)c, n, out);
  return done("to_fp64");
}
int launch_from_fp64(const double* in, int64_t n, int precision, void* hi, void* c, cudaStream_t s) {
  if (precision == LAT_FP64) from64_kernel<double, false><<<grid_for(n), 256, 0, s>>>(in, n, (double*)hi, nullptr);
  else from64_kernel<float, true><<<grid_for(n), 256, 0, s>>>(in, n, (float*)hi, (float*)c);
  return done("from_fp64");
}

int launch_vacuum_modes(const VacArgs& a, cudaStream_t s) {
  const int64_t M = (int64_t)(a.nx / 2 + 1) * a.ny * a.nz;
  vacuum_kernel<<<grid_for(M), 256, 0, s>>>(a);
  return done("vacuum");
}
int launch_fd_laplacian64(const double* in, double* out, int nx, int ny, int nz, const double* lc, cudaStream_t s) {
  fd_lap64_kernel<<<grid_for((int64_t)nx * ny * nz), 256, 0, s>>>(in, out, nx, ny, nz, lc[0], lc[1], lc[2], lc[3]);
  return done("fd laplacian");
}
int launch_sample_steps(int step, const SampleArgs& a, cudaStream_t s) {
  const int blk = 256;
  auto grid = [&](int64_t n) { return (unsigned)std::min<int64_t>((n + blk - 1) / blk, 4096); };
  switch (step) {
    case 0: sample_dst_in_kernel<<<grid(4LL * a.nos), blk, 0, s>>>(a.z, a.nos, a.dkos, a.m2, a.gamma, a.kcut); break;
    case 1: sample_dst_out_kernel<<<grid(a.nos), blk, 0, s>>>(a.z, a.nos, a.norm, a.ker); break;
    case 2: sample_kernel3d<<<grid((int64_t)a.n * a.n * a.n), blk, 0, s>>>(a.ker, a.n, a.f); break;
    case 3: sample_noise_kernel<<<grid(a.M), blk, 0, s>>>(a.F, a.M, a.seed, a.stream); break;
    case 4: sample_hermitize_kernel<<<grid(2LL * a.n * a.n), blk, 0, s>>>(a.F, a.n); break;
    default: return set_error(LAT_ERR_ARG, "sample step");
  }
  if (g_launch_counter) ++*g_launch_counter;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, "sample launch");
}

int launch_add_scale(double* f, int64_t n, double scale, double offset, cudaStream_t s) {
  add_scale_kernel<<<grid_for(n), 256, 0, s>>>(f, n, scale, offset);
  return done("add_scale");
}
int launch_bubbles(double* phi, int nx, int ny, int nz, double dx, int nbub, const double* cen, double R, double w,
                   cudaStream_t s) {
  bubbles_kernel<<<grid_for((int64_t)nx * ny * nz), 256, 0, s>>>(phi, nx, ny, nz, dx, nbub, cen, R, w);
  return done("bubbles");
}

}  // namespace lat
