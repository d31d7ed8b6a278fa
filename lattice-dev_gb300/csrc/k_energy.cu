// k_energy.cu -- lattice sums of the energy output.
//
// dump_rho (Pseudospec/openmp_dev/evolve_spectral.f90:305-415) and homlat's
// grad_en, grad_en_wlap, pot_en, kinetic_en (Discrete/Bubble-Collisions/
// homlat.f90:65-188).  The sums of an FP64 lattice are bound by the FP64 pipe
// (2 operations per clock and SM), those of a small one by latency: every
// kernel takes only the sums its lattice needs, few enough blocks that the
// reduction does not outweigh them, and each stencil value once.
#include <algorithm>

#include "engine.hpp"

namespace lat {

namespace {

inline int done(const char* what) {
  if (g_launch_counter) ++*g_launch_counter;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? LAT_OK : cuda_fail(e, what);
}

// ------------------------------------------- sums of one site at a time
// sum pi^2, V, phi_1, phi_2 over sites [t, tend) in steps of `step`
template <typename R, int NF, typename Acc>
__device__ __forceinline__ void site_sums(const R* phi, const R* pi, int64_t fs, int64_t t, int64_t tend, int64_t step,
                                          const ModelP& m, Acc (&s)[4]) {
  for (; t < tend; t += step) {
    R f[NF];
#pragma unroll
    for (int l = 0; l < NF; ++l) {
      f[l] = phi[l * fs + t];
      const R p = pi[l * fs + t];
      s[0].add(p * p);
    }
    s[1].add(model_v<R, NF>(m, f));
    s[2].add(f[0]);
    if (NF > 1) s[3].add(f[NF - 1]);
  }
}

// four sites per access (16-byte aligned arrays whose length is a multiple of four)
template <typename R> struct Quad;
template <> struct Quad<float> {
  static __device__ __forceinline__ void ld(const float* p, float (&v)[4]) {
    const float4 t = __ldcs(reinterpret_cast<const float4*>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  }
};
template <> struct Quad<double> {
  static __device__ __forceinline__ void ld(const double* p, double (&v)[4]) {
    const double2 a = __ldcs(reinterpret_cast<const double2*>(p)), b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
};
template <typename R, int NF, typename Acc>
__device__ __forceinline__ void quad_sums(const R* phi, const R* pi, int64_t fs, int64_t q, int64_t qend, int64_t step,
                                          const ModelP& m, Acc (&s)[4]) {
  for (; q < qend; q += step) {
    R f4[NF][4], p4[NF][4];
#pragma unroll
    for (int l = 0; l < NF; ++l) {
      Quad<R>::ld(phi + l * fs + 4 * q, f4[l]);
      Quad<R>::ld(pi + l * fs + 4 * q, p4[l]);
    }
    R ke = R(0), pe = R(0), m0 = R(0), m1 = R(0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      R f[NF];
#pragma unroll
      for (int l = 0; l < NF; ++l) {
        f[l] = f4[l][j];
        ke += p4[l][j] * p4[l][j];
      }
      pe += model_v<R, NF>(m, f);
      m0 += f[0];
      if (NF > 1) m1 += f[NF - 1];
    }
    s[0].add(ke);
    s[1].add(pe);
    s[2].add(m0);
    if (NF > 1) s[3].add(m1);
  }
}

// Spectral lattices: red[0..3]
template <typename R, int NF>
__global__ void __launch_bounds__(256) energy_kernel(EnergyArgs a) {
  using Acc = typename AccOf<R>::type;
  Acc s[4];
  const int64_t N = (int64_t)a.nx * a.ny * a.nz;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  const R *phi = static_cast<const R*>(a.phi), *pi = static_cast<const R*>(a.pi);
  if (N % 4 == 0) quad_sums<R, NF>(phi, pi, N, t0, N / 4, step, a.model, s);
  else site_sums<R, NF>(phi, pi, N, t0, N, step, a.model, s);
  const typename Acc::Red v[4] = {s[0].red(), s[1].red(), s[2].red(), s[3].red()};
  double tot[4];
  if (grid_reduce<4>(v, a.rb, tot)) {
    for (int i = 0; i < 4; ++i) {
      a.sc->red[i] = tot[i];
      if (bad(tot[i])) a.sc->err |= 1u;
    }
  }
}

// ------------------------------------------------------------- stencils
// FP64 finite-difference lattices: red[0..3], red[4] = -sum phi L phi, red[5] = sum
// of the squared differences and, with strains, red[6] = sum w pu^2, red[7] =
// -sum w u L u (w = 2 off the diagonal), over planes [zlo, zhi).  A thread
// marches along z and reads a plane once (9 values instead of 27 per site); per
// array it keeps what the last plane adds to its neighbours and the Laplacian in
// progress, as the FP64 steps do.  Each pair of neighbours enters the squared
// differences once, at its lower site, for both.  Bound by the FP64 pipe.
template <int NF, bool GW, bool SEVEN>
__global__ void __launch_bounds__(128) fd_energy_kernel(EnergyArgs a, int zlo, int zhi, int zc) {
  using R = double;
  constexpr int NC = NF + (GW ? 6 : 0);
  using Acc = typename AccOf<R>::type;
  Acc s[8];
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int64_t N = (int64_t)nx * ny * nz, plane = (int64_t)nx * ny;
  const int gx = (nx + 31) / 32;  // tiles of 32 x 4 sites, row by row along the grid's x
  const int x = (int)(blockIdx.x % gx) * 32 + threadIdx.x, y = (int)(blockIdx.x / gx) * 4 + threadIdx.y;
  const int z0 = zlo + blockIdx.z * zc, z1 = min(z0 + zc, zhi);
  if (x < nx && y < ny) {
    const int xm = x ? x - 1 : nx - 1, xp = x + 1 < nx ? x + 1 : 0;
    const int row[3] = {(y ? y - 1 : ny - 1) * nx, y * nx, (y + 1 < ny ? y + 1 : 0) * nx};
    const R c0 = (R)a.c[0], c1 = (R)a.c[1], c2 = (R)a.c[2], c3 = (R)a.c[3];
    auto wrap = [&](int z) { return z < 0 ? z + nz : (z >= nz ? z - nz : z); };
    auto base = [&](int c) {
      return c < NF ? static_cast<const R*>(a.phi) + c * N : static_cast<const R*>(a.u) + (c - NF) * N;
    };
    R wc[NC][3], tz[NC], la[NC], ln[NC];  // centres; neighbour term; Laplacian of planes z, z + 1
    R e1[NF], e2[NF];  // in-plane squared differences of the middle plane's pairs
    // plane z into slot k; diffs of the pairs (z-1, z) and inside z for the fields
    auto load = [&](int z, int k, bool pairs) {
      const int64_t zo = (int64_t)wrap(z) * plane;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const R* g = base(c) + zo;
        R v[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          v[j][1] = __ldg(g + row[j] + x);
          if (!SEVEN || j == 1) {
            v[j][0] = __ldg(g + row[j] + xm);
            v[j][2] = __ldg(g + row[j] + xp);
          }
        }
        wc[c][k] = v[1][1];
        const R s1 = (v[1][0] + v[1][2]) + (v[0][1] + v[2][1]);
        const R s2 = SEVEN ? R(0) : (v[0][0] + v[0][2]) + (v[2][0] + v[2][2]);
        const R t = SEVEN ? c1 * v[1][1] : c1 * v[1][1] + c2 * s1 + c3 * s2;
        if (k == 2) la[c] += t;  // plane z - 1 is complete
        if (k > 0) ln[c] = SEVEN ? tz[c] + c0 * v[1][1] + c1 * s1 : tz[c] + c0 * v[1][1] + c1 * s1 + c2 * s2;
        if (k == 1) la[c] = ln[c];
        tz[c] = t;
        if (c < NF) {
          auto sq = [](R p, R q) { const R d = p - q; return d * d; };
          if (pairs) {  // with plane z - 1 (slot k - 1)
            const R o = wc[c][k - 1];
            R q1 = sq(v[1][1], o) + e1[c], q2 = R(0), q3 = R(0);
            if (!SEVEN) {
              q2 = ((sq(v[1][0], o) + sq(v[1][2], o)) + (sq(v[0][1], o) + sq(v[2][1], o))) + e2[c];
              q3 = (sq(v[0][0], o) + sq(v[0][2], o)) + (sq(v[2][0], o) + sq(v[2][2], o));
            }
            R t = c1 * q1;
            if (!SEVEN) t += c2 * q2 + c3 * q3;
            s[5].add(t + t);
          }
          e1[c] = sq(v[1][2], v[1][1]) + sq(v[2][1], v[1][1]);
          if (!SEVEN) e2[c] = sq(v[2][2], v[1][1]) + sq(v[2][0], v[1][1]);
        }
      }
    };
    load(z0 - 1, 0, false);
    load(z0, 1, false);
    for (int z = z0; z < z1; ++z) {
      const int64_t t = (int64_t)z * plane + row[1] + x;
      load(z + 1, 2, true);
      R f[NF], ke = R(0);
#pragma unroll
      for (int l = 0; l < NF; ++l) {
        f[l] = wc[l][1];
        const R p = static_cast<const R*>(a.pi)[l * N + t];
        ke += p * p;
        s[4].add(-f[l] * la[l]);
      }
      s[0].add(ke);
      s[1].add(model_v<R, NF>(a.model, f));
      s[2].add(f[0]);
      if (NF > 1) s[3].add(f[NF - 1]);
      if (GW) {
        R d = R(0), o = R(0), dl = R(0), ol = R(0);
#pragma unroll
        for (int g = 0; g < 6; ++g) {
          const R p = static_cast<const R*>(a.pu)[g * N + t];
          if (g < 3) { d += p * p; dl -= wc[NF + g][1] * la[NF + g]; }
          else { o += p * p; ol -= wc[NF + g][1] * la[NF + g]; }
        }
        s[6].add(d + (o + o));
        s[7].add(dl + (ol + ol));
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        wc[c][0] = wc[c][1];
        wc[c][1] = wc[c][2];
        la[c] = ln[c];
      }
    }
  }
  constexpr int NV = GW ? 8 : 6;
  typename Acc::Red v[NV];
  double tot[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = s[i].red();
  if (grid_reduce<NV>(v, a.rb, tot)) {
    for (int i = 0; i < NV; ++i) {
      a.sc->red[i] = tot[i];
      if (bad(tot[i])) a.sc->err |= 1u;
    }
    for (int i = NV; i < 8; ++i) a.sc->red[i] = 0.0;
  }
}

// The same sums of FP32 lattices.  An FP32 term's rounding is part of the
// result (1e-9 of an energy), so every site's neighbours are added in the order
// of the reference's loops; a thread keeps three planes of one array's 3 x 3
// values (9 reads a site instead of 27) and takes the arrays one after another.
template <int NF, bool GW, bool SEVEN>
__global__ void __launch_bounds__(128) fd_energy32_kernel(EnergyArgs a, int zlo, int zhi, int zc) {
  using R = float;
  constexpr int NC = NF + (GW ? 6 : 0);
  KSum s[8];
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int64_t N = (int64_t)nx * ny * nz, plane = (int64_t)nx * ny;
  const int gx = (nx + 31) / 32;  // tiles of 32 x 4 sites, row by row along the grid's x
  const int x = (int)(blockIdx.x % gx) * 32 + threadIdx.x, y = (int)(blockIdx.x / gx) * 4 + threadIdx.y;
  const int z0 = zlo + blockIdx.z * zc, z1 = min(z0 + zc, zhi);
  if (x < nx && y < ny) {
    const int col[3] = {x ? x - 1 : nx - 1, x, x + 1 < nx ? x + 1 : 0};
    const int row[3] = {(y ? y - 1 : ny - 1) * nx, y * nx, (y + 1 < ny ? y + 1 : 0) * nx};
    const R c0 = (R)a.c[0], c1 = (R)a.c[1], c2 = (R)a.c[2], c3 = (R)a.c[3];
    auto wrap = [&](int z) { return z < 0 ? z + nz : (z >= nz ? z - nz : z); };
#pragma unroll 1
    for (int c = 0; c < NC; ++c) {
      const R* g = c < NF ? static_cast<const R*>(a.phi) + c * N : static_cast<const R*>(a.u) + (c - NF) * N;
      R v[3][3][3];
      auto load = [&](int z, R (&w)[3][3]) {
        const R* gz = g + (int64_t)wrap(z) * plane;
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int i = 0; i < 3; ++i)
            if (!SEVEN || i == 1 || j == 1) w[j][i] = __ldg(gz + row[j] + col[i]);
      };
      load(z0 - 1, v[0]);
      load(z0, v[1]);
      for (int z = z0; z < z1; ++z) {
        load(z + 1, v[2]);
        const int64_t t = (int64_t)z * plane + row[1] + x;
        const R g0 = v[1][1][1];
        R r1 = 0, r2 = 0, r3 = 0, q1 = 0, q2 = 0, q3 = 0;
#pragma unroll
        for (int dz = 0; dz < 3; ++dz)
#pragma unroll
          for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
              const int rank = (dx != 1) + (dy != 1) + (dz != 1);
              if (rank == 0 || (SEVEN && rank > 1)) continue;
              const R w = v[dz][dy][dx], d = w - g0;
              if (rank == 1) { r1 += w; q1 += d * d; }
              else if (rank == 2) { r2 += w; q2 += d * d; }
              else { r3 += w; q3 += d * d; }
            }
        const R lapsum = c0 * g0 + c1 * r1 + c2 * r2 + c3 * r3;
        if (c < NF) {
          const R grad2 = c1 * q1 + c2 * q2 + c3 * q3;
          const R p = static_cast<const R*>(a.pi)[c * N + t];
          s[0].add(p * p);
          s[4].add(-g0 * lapsum);
          s[5].add(grad2);
          if (c == 0) {
            R f[NF];
            f[0] = g0;
            if (NF > 1) f[NF - 1] = static_cast<const R*>(a.phi)[(NF - 1) * N + t];
            s[1].add(model_v<R, NF>(a.model, f));
            s[2].add(f[0]);
            if (NF > 1) s[3].add(f[NF - 1]);
          }
        } else {
          const R w = c - NF < 3 ? R(1) : R(2);
          const R p = static_cast<const R*>(a.pu)[(c - NF) * N + t];
          s[6].add(w * p * p);
          s[7].add(-w * g0 * lapsum);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            v[0][j][i] = v[1][j][i];
            v[1][j][i] = v[2][j][i];
          }
      }
    }
  }
  constexpr int NV = GW ? 8 : 6;
  FF v[NV];
  double tot[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = s[i].red();
  if (grid_reduce<NV>(v, a.rb, tot)) {
    for (int i = 0; i < NV; ++i) {
      a.sc->red[i] = tot[i];
      if (bad(tot[i])) a.sc->err |= 1u;
    }
    for (int i = NV; i < 8; ++i) a.sc->red[i] = 0.0;
  }
}

// LOG.out's ball: over the sites with |(x, y, z) + 1 - n/2|^2 dx^2 < ball_r2
// (1-based indices about n/2, iofile.f90:552) red[9] = sum (sum_f pi_f)^2,
// red[10] = the stencil's gradient squared, red[11] = V
template <typename R, int NF>
__global__ void __launch_bounds__(256) ball_kernel(EnergyArgs a) {
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int64_t N = (int64_t)nx * ny * nz;
  const R *phi = static_cast<const R*>(a.phi), *pi = static_cast<const R*>(a.pi);
  using Acc = typename AccOf<R>::type;
  Acc s[3];
  const R c[3] = {(R)a.c[1], (R)a.c[2], (R)a.c[3]};
  auto wrapi = [](int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); };
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(t % nx), y = (int)((t / nx) % ny), z = (int)(t / ((int64_t)nx * ny));
    const double bx = x + 1 - nx / 2, by = y + 1 - ny / 2, bz = z + 1 - nz / 2;
    if (!((bx * bx + by * by + bz * bz) * a.dx * a.dx < a.ball_r2)) continue;
    R f[NF], psum = R(0), g2 = R(0);
#pragma unroll
    for (int l = 0; l < NF; ++l) {
      const R* g = phi + l * N;
      f[l] = g[t];
      psum += pi[l * N + t];
      R q[3] = {R(0), R(0), R(0)};
      for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
          for (int dx = -1; dx <= 1; ++dx) {
            const int rank = (dx != 0) + (dy != 0) + (dz != 0);
            if (rank == 0) continue;
            const R d = g[((int64_t)wrapi(z + dz, nz) * ny + wrapi(y + dy, ny)) * nx + wrapi(x + dx, nx)] - f[l];
            q[rank - 1] += d * d;
          }
      g2 += c[0] * q[0] + c[1] * q[1] + c[2] * q[2];
    }
    s[0].add(psum * psum);
    s[1].add(g2);
    s[2].add(model_v<R, NF>(a.model, f));
  }
  const typename Acc::Red v[3] = {s[0].red(), s[1].red(), s[2].red()};
  double tot[3];
  if (grid_reduce<3>(v, a.rb, tot)) {
    for (int i = 0; i < 3; ++i) {
      a.sc->red[9 + i] = tot[i];
      if (bad(tot[i])) a.sc->err |= 1u;
    }
  }
}

template <typename R, int NF>
int energy_go(const EnergyArgs& a, cudaStream_t s) {
  const int64_t N = (int64_t)a.nx * a.ny * a.nz;
  if (!a.fd) {
    // eight sites a thread, at most three blocks an SM
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(a.grid * 3 / 4, (N + 2047) / 2048));
    energy_kernel<R, NF><<<grid, 256, 0, s>>>(a);
    return done("energy");
  }
  const int64_t plane = (int64_t)a.nx * a.ny;
  const int zlo = a.t_hi > 0 ? (int)(a.t_lo / plane) : 0, zhi = a.t_hi > 0 ? (int)(a.t_hi / plane) : a.nz;
  const bool seven = a.c[2] == 0.0 && a.c[3] == 0.0;
  // planes per block: two planes are read beyond each chunk, so as few chunks
  // as give every SM eight blocks (144 x 100 x 90 GW FP64: 784 us with two)
  const int gx = (a.nx + 31) / 32, gy = (a.ny + 3) / 4;
  const int want = std::max(1, (8 * (a.grid / 4) + gx * gy - 1) / (gx * gy));
  const int zc = std::max(2, (zhi - zlo + want - 1) / want);
  const dim3 grid(gx * gy, 1, (zhi - zlo + zc - 1) / zc), block(32, 4);
#define LAT_FD_ENERGY(GWV, SEV)                                                                          \
  do {                                                                                                  \
    if constexpr (sizeof(R) == 8) fd_energy_kernel<NF, GWV, SEV><<<grid, block, 0, s>>>(a, zlo, zhi, zc); \
    else fd_energy32_kernel<NF, GWV, SEV><<<grid, block, 0, s>>>(a, zlo, zhi, zc);                        \
  } while (0)
  if (a.u) {
    if (seven) LAT_FD_ENERGY(true, true);
    else LAT_FD_ENERGY(true, false);
  } else {
    if (seven) LAT_FD_ENERGY(false, true);
    else LAT_FD_ENERGY(false, false);
  }
#undef LAT_FD_ENERGY
  const int st = done("energy");
  if (st != LAT_OK || !(a.ball_r2 > 0.0)) return st;
  ball_kernel<R, NF><<<a.grid, 256, 0, s>>>(a);
  return done("ball energy");
}

// ------------------------------------------------------------- Parseval
// Sum over a half spectrum of w k^2 |F_k|^2, w = 2 for the modes whose
// conjugate partner is not stored.  A warp takes the (up to four) rows (+-y,
// +-z), which share k_y^2 + k_z^2, together.  FP64 adds them before two
// multiply-adds; in FP32 every mode's term enters the compensated sum by itself.
template <typename R, typename C, typename Acc>
__device__ __forceinline__ void parseval_rows(const C* F, int nx, int ny, int nz, R dkx2, double dky2, double dkz2,
                                              int row0, int step, int lane, Acc& acc) {
  const int hx = nx / 2 + 1, hy = ny / 2 + 1, hz = nz / 2 + 1;
  for (int row = row0; row < hy * hz; row += step) {
    const int jj = row % hy, kk = row / hy;
    const R kyz = (R)((double)((int64_t)jj * jj) * dky2 + (double)((int64_t)kk * kk) * dkz2);
    const int my = (jj == 0 || 2 * jj == ny) ? 1 : 2, mz = (kk == 0 || 2 * kk == nz) ? 1 : 2;
    size_t at[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int y = my == 2 && (r & 1) ? ny - jj : jj, z = (my == 2 ? r >> 1 : r) ? nz - kk : kk;
      at[r] = ((size_t)z * ny + y) * hx;
    }
#pragma unroll 2
    for (int x = lane; x < hx; x += 32) {
      C v[4];  // in flight together
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        v[r] = C{0, 0};
        if (r < my * mz) v[r] = F[at[r] + x];
      }
      const bool twice = x != 0 && 2 * x != nx;
      R k2 = (R)((int64_t)x * x) * dkx2 + kyz;
      if constexpr (sizeof(R) == sizeof(double)) {
        R t = R(0);
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (r < my * mz) t += v[r].x * v[r].x + v[r].y * v[r].y;
        if (twice) t += t;
        acc.add(k2 * t);
      } else {
        if (twice) k2 += k2;
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (r < my * mz) acc.add(k2 * (v[r].x * v[r].x + v[r].y * v[r].y));
      }
    }
  }
}

template <typename R, typename C>
__global__ void __launch_bounds__(256) parseval_kernel(const C* F, int nx, int ny, int nz, int nf, double dkx2,
                                                       double dky2, double dkz2, DevScalars* sc, int slot,
                                                       RedBuf rb) {
  using Acc = typename AccOf<R>::type;
  Acc acc;
  const size_t M = (size_t)(nx / 2 + 1) * ny * nz;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int l = 0; l < nf; ++l)
    parseval_rows<R>(F + l * M, nx, ny, nz, (R)dkx2, dky2, dkz2, warp, nwarp, threadIdx.x & 31, acc);
  const typename Acc::Red v[1] = {acc.red()};
  double t[1];
  if (grid_reduce<1>(v, rb, t)) sc->red[slot] = t[0];
}

// ------------------------------------------------------------- ensembles
// Every run of an ensemble in one launch: blockIdx.x is the run (along y a grid
// holds 65535 blocks, an ensemble may hold more runs), its first run.blocks
// blocks share it; the last to arrive leaves the run's sums in out[run * 8 ..]
// in block order.  MODE 0: sum pi^2, V, phi; 1: Parseval sum.
template <typename R, typename C, int MODE>
__global__ void __launch_bounds__(256) ens_energy_kernel(EnsEnergyArgs a) {
  constexpr int NV = MODE == 0 ? 3 : 1;
  __shared__ int am_last;
  const EnsEnergyRun run = a.runs[blockIdx.x];
  const int n = run.n, nblk = run.blocks;
  if ((int)blockIdx.y >= nblk) return;
  using Acc = typename AccOf<R>::type;
  double s[NV];
  if (MODE == 0) {
    Acc q[4];
    const int64_t N = (int64_t)n * n * n;
    const R *phi = static_cast<const R*>(a.phi) + run.site, *pi = static_cast<const R*>(a.pi) + run.site;
    const int64_t t0 = (int64_t)blockIdx.y * blockDim.x + threadIdx.x, step = (int64_t)nblk * blockDim.x;
    if (N % 4 == 0 && run.site % 4 == 0) quad_sums<R, 1>(phi, pi, N, t0, N / 4, step, a.model, q);
    else site_sums<R, 1>(phi, pi, N, t0, N, step, a.model, q);
    const typename Acc::Red v[3] = {q[0].red(), q[1].red(), q[2].red()};
    double b[3];
    block_sums<3>(v, b);
    for (int i = 0; i < NV; ++i) s[i] = b[i];
  } else {
    Acc acc;
    const int warp = (blockIdx.y * blockDim.x + threadIdx.x) >> 5, nwarp = (nblk * blockDim.x) >> 5;
    parseval_rows<R>(static_cast<const C*>(a.Fk) + run.fk, n, n, n, (R)run.dk2, run.dk2, run.dk2, warp, nwarp,
                     threadIdx.x & 31, acc);
    const typename Acc::Red v[1] = {acc.red()};
    double b[1];
    block_sums<1>(v, b);
    s[0] = b[0];
  }
  double* part = a.partials + (size_t)blockIdx.x * a.max_blocks * 4;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NV; ++i) part[(size_t)blockIdx.y * NV + i] = s[i];
    __threadfence();
    am_last = atomicAdd(a.counters + blockIdx.x, 1u) == (unsigned int)nblk - 1u;
  }
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  double tot[NV];
  row_sums<NV>(part, nblk, tot);
  if (threadIdx.x == 0) {
    for (int i = 0; i < NV; ++i) a.out[(size_t)blockIdx.x * 8 + (MODE == 0 ? i : 4)] = tot[i];
    a.counters[blockIdx.x] = 0u;
  }
}

}  // namespace

int launch_energy(const EnergyArgs& a, int precision, cudaStream_t s) {
  if (a.nf == 1) return precision == LAT_FP64 ? energy_go<double, 1>(a, s) : energy_go<float, 1>(a, s);
  if (a.nf == 2) return precision == LAT_FP64 ? energy_go<double, 2>(a, s) : energy_go<float, 2>(a, s);
  return set_error(LAT_ERR_UNSUPPORTED, "energies support nfld = 1 or 2");
}

int launch_parseval(const void* Fk, int nx, int ny, int nz, int nf, double dkx2, double dky2, double dkz2,
                    DevScalars* sc, int slot, RedBuf rb, int grid, int precision, cudaStream_t s) {
  // a warp per row; at most `grid` blocks
  const int rows = (ny / 2 + 1) * (nz / 2 + 1);
  grid = std::max(1, std::min(grid, (rows + 7) / 8));
  if (precision == LAT_FP64)
    parseval_kernel<double, double2><<<grid, 256, 0, s>>>((const double2*)Fk, nx, ny, nz, nf, dkx2, dky2, dkz2, sc, slot, rb);
  else
    parseval_kernel<float, float2><<<grid, 256, 0, s>>>((const float2*)Fk, nx, ny, nz, nf, dkx2, dky2, dkz2, sc, slot, rb);
  return done("parseval");
}

int launch_ens_energies(const EnsEnergyArgs& a, int nruns, int parseval, int precision, cudaStream_t s) {
  const dim3 grid(nruns, a.max_blocks);  // at most 64 blocks a run
  if (precision == LAT_FP64) {
    if (parseval) ens_energy_kernel<double, double2, 1><<<grid, 256, 0, s>>>(a);
    else ens_energy_kernel<double, double2, 0><<<grid, 256, 0, s>>>(a);
  } else {
    if (parseval) ens_energy_kernel<float, float2, 1><<<grid, 256, 0, s>>>(a);
    else ens_energy_kernel<float, float2, 0><<<grid, 256, 0, s>>>(a);
  }
  return done("ensemble energies");
}

}  // namespace lat
