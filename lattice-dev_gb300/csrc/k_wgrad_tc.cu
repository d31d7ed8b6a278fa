// k_wgrad_tc.cu -- weight gradients of the closure's layers with 32 input
// channels on the 5th-generation tensor cores.
//
//   dW[tap][i][o] = sum over sites s of X[s + off(tap)][i] D[s][o]
//
// The sites are K.  A K16 step is 16 consecutive x of one row.  M = 128 is four
// consecutive halo rows (dy 0, 1, 2 and one unused) of 32 input channels of one
// X plane; N is the output channels of the three D planes that meet it (tap
// planes 2, 1, 0; 96 columns, or 32 with 8 unused ones), so three MMAs, one for
// each dx, give all 27 taps.  Their accumulators stay in tensor memory for the
// whole kernel; a block writes one partial sum per weight at its end.
//
// Both operands are read from the channels-last arrays as they are, M (or N)
// along the 16 bytes of a core matrix (8 channels x 8 sites, no swizzle):
//   X: halo plane [row 10][chunk 4][x 34][8 channels], a ring of three; the 16
//      core matrices of the four rows sit at one stride, a tap's x offset is a
//      16-byte shift;
//   D: [plane][chunk][site 256][8 channels], a ring of six planes whose first
//      two are kept twice, behind the sixth, so that any three planes in a row
//      are one operand.  Planes outside the block's run are zeros.
// A step is one X plane of 32 x 8 sites (48 MMAs); blocks take equal runs of
// planes, column by column, and march through z.  Eight warps issue copies,
// wait for the MMAs and add the columns of D (the biases); one warp,
// converged, issues the MMAs.
//
// Four 64^3 lattices, 32 x 32 and 32 x 8 channels: 222 and 107 us by mma.sync
// (that instruction's rate bounds it), 155 and 94 with one MMA per (dz, dx) of
// N = 32 or 16, 91 and 44 so.  Left: the copies of 34 x 10 positions for 32 x 8
// sites and a block barrier a step.
#include <cuda_bf16.h>
#include <stdint.h>

#include <algorithm>

#include "net.hpp"
#include "tc.cuh"

namespace lat {
namespace net {

namespace {

constexpr int WX = 32, WY = 8, PX = WX + 2, PY = WY + 2;  // sites of a step, of its halo plane
constexpr int CHX = PX * 16, ROWX = 4 * CHX, PLANEX = PY * ROWX;
constexpr int NX = 3, ND = 6;            // rings of X and D planes
constexpr int NPX = (PY * PX * 4 + 255) / 256;  // copies of an X plane per thread
constexpr int CHD = WX * WY * 16;        // bytes per 8-channel chunk of D
constexpr int WWORK = 256, WTHREADS = WWORK + 32, WMMA = WWORK / 32;
constexpr int WTMEM = 512;               // three accumulators of 96 columns

template <int CD>
struct WgGeom {
  static constexpr int CH = CD / 8;
  static constexpr int DSLOT = CH * CHD;
  static constexpr int XB = NX * PLANEX;
  static constexpr int N = CD == 8 ? 32 : 96;
  // CD 8: a fourth plane is read with the last three (and its columns ignored)
  static constexpr int SMEM = XB + (ND + 2 + (CD == 8 ? 1 : 0)) * DSLOT + 64;
  static_assert(ROWX <= DSLOT, "the unused row behind the last plane is inside the block's memory");
};

// kind::f16, A and B BF16, D FP32, both with M (N) along the 16 bytes, M = 128
template <int N>
constexpr uint32_t wg_idesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
}

template <int CD>
__global__ void __launch_bounds__(WTHREADS, 1) wgrad_tc_kernel(WgradArgs a, int* err) {
  using G = WgGeom<CD>;
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* tail = sm + G::SMEM - 64;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(tail);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(tail + 32);
  volatile int* abort = reinterpret_cast<volatile int*>(tail + 48);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t x_s = su32(sm), d_s = x_s + G::XB;
  const uint32_t mb[2] = {su32(mbar), su32(mbar + 1)};
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(su32(tslot)), "r"(WTMEM));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  if (tid == 0) {
    *abort = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mb[0]));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mb[1]));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);

  const int tiles_x = a.nx / WX, cols_per = tiles_x * (a.ny / WY);
  const int64_t nsteps = (int64_t)cols_per * a.nlat * a.nz, Nsite = (int64_t)a.nx * a.ny * a.nz;
  uint32_t phase[2] = {0, 0};
  int pending[2] = {0, 0};  // commits not yet waited for
  bool failed = false, first = true;
  float bs[8];  // sums of 8 channels of D
#pragma unroll
  for (int k = 0; k < 8; ++k) bs[k] = 0.f;

  uint32_t soff[NPX];  // this thread's copies of an X plane: places in a ring slot
#pragma unroll
  for (int l = 0; l < NPX; ++l) {
    const int i = tid + l * WWORK, hx = (i >> 2) % PX, hy = (i >> 2) / PX;
    soff[l] = hy * ROWX + (i & 3) * CHX + hx * 16;
  }
  int64_t st = nsteps * blockIdx.x / gridDim.x;
  const int64_t st_end = nsteps * (blockIdx.x + 1) / gridDim.x;
  while (st < st_end && !failed) {
    const int64_t col = st / a.nz;
    const int zA = (int)(st % a.nz);
    const int nzs = (int)min((int64_t)(a.nz - zA), st_end - st);
    st += nzs;
    const int64_t li = col / cols_per;
    const int cr = (int)(col % cols_per);
    const int x0 = cr % tiles_x * WX, y0 = cr / tiles_x * WY;
    const __nv_bfloat16 *X = a.x + li * Nsite * 32, *D = a.d + li * Nsite * CD;
    int goff[NPX];
#pragma unroll
    for (int l = 0; l < NPX; ++l) {
      const int i = tid + l * WWORK, hx = (i >> 2) % PX, hy = (i >> 2) / PX;
      int x = x0 + hx - 1, y = y0 + hy - 1;
      x = x < 0 ? x + a.nx : (x >= a.nx ? x - a.nx : x);
      y = y < 0 ? y + a.ny : (y >= a.ny ? y - a.ny : y);
      goff[l] = (y * a.nx + x) * 32 + (i & 3) * 8;
    }
    const int nin = nzs + 2;
    // D plane zA + u - 2 (u = 0 .. nin + 1) into slot u % 6 and, of the first two, its copy
    auto load_d = [&](int u) {
      const int q = u - 2, slot = u % ND;
      const __nv_bfloat16* src = D + ((int64_t)(zA + q) * a.ny + y0) * a.nx * CD + (int64_t)x0 * CD;
#pragma unroll
      for (int c = 0; c < (slot < 2 ? 2 : 1); ++c) {
        const uint32_t base = G::XB + (slot + c * ND) * G::DSLOT;
        for (int i = tid; i < WX * WY * G::CH; i += WWORK) {
          const int ch = i % G::CH, s = i / G::CH;
          const uint32_t dst = base + ch * CHD + s * 16;
          if (q >= 0 && q < nzs) cp16(x_s + dst, src + ((int64_t)(s / WX) * a.nx + s % WX) * CD + ch * 8);
          else *reinterpret_cast<uint4*>(sm + dst) = make_uint4(0, 0, 0, 0);
        }
      }
    };
    // X plane zA + t - 1 into slot t % 3, the last D plane that step t takes
    auto load = [&](int t) {
      if (t < nin && warp != WMMA) {
        int z = zA + t - 1;
        z = z < 0 ? z + a.nz : (z >= a.nz ? z - a.nz : z);
        const __nv_bfloat16* pl = X + (int64_t)z * a.ny * a.nx * 32;
        const uint32_t base = x_s + t % NX * PLANEX;
#pragma unroll
        for (int l = 0; l < NPX; ++l)
          if (l + 1 < NPX || tid + l * WWORK < PY * PX * 4) cp16(base + soff[l], pl + goff[l]);
        load_d(t + 2);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (warp != WMMA) {
      load_d(0);
      load_d(1);
    }
    load(0);
    load(1);
#pragma unroll 1
    for (int t = 0; t <= nin; ++t) {
      const int buf = t & 1;
      if (t < nin) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (*abort) {  // read after the barrier: every thread sees the same value
          failed = true;
          break;
        }
        if (warp == WMMA) {
          const uint32_t lead = elect_lane();
          const uint64_t bd0 = mdesc(d_s + t % ND * G::DSLOT, 128, CHD);
          const uint64_t ad0 = mdesc(x_s + t % NX * PLANEX, 128, CHX);
          const uint32_t acc0 = first ? 0u : 1u;
          first = false;
#pragma unroll
          for (int ks = 0; ks < WY * WX / 16; ++ks) {
            const int r = ks / (WX / 16), kx = ks % (WX / 16);
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
              mma_bf16(lead, tmem + dx * G::N, ad0 + (uint64_t)((r * ROWX + (kx * 16 + dx) * 16) >> 4),
                       bd0 + (uint64_t)(ks * 256 >> 4), wg_idesc<G::N>(), ks == 0 ? acc0 : 1u);
          }
          asm volatile(
              "{\n .reg .pred e;\n setp.ne.b32 e, %1, 0;\n"
              " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(mb[buf]),
              "r"(lead)
              : "memory");
          __syncwarp();
        } else {  // bias sums of plane u = t + 2: chunk tid % CH, every (256 / CH)-th site
          const uint4* dp = reinterpret_cast<const uint4*>(sm + G::XB + (t + 2) % ND * G::DSLOT + tid % G::CH * CHD);
#pragma unroll
          for (int s = 0; s < G::CH; ++s) {
            const uint4 v = dp[tid / G::CH + s * (WWORK / G::CH)];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              bs[2 * k] += __uint_as_float(w[k] << 16);
              bs[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
            }
          }
        }
        pending[buf] = 1;
      }
      if (t >= 1 && warp != WMMA) {
        const int pb = buf ^ 1;
        uint32_t spins = 0;
        int to = 0;
        while (!mbar_try(mb[pb], phase[pb])) {
          if (++spins > kSpinLimit) {
            to = 1;
            break;
          }
        }
        if (__any_sync(0xffffffffu, to)) {
          if (lane == 0) *abort = 1;
        } else {
          phase[pb] ^= 1u;
          pending[pb] = 0;
        }
      }
      load(t + 2);  // X into the slot that step t - 1 read
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if (*abort) failed = true;
  }
  if (failed) {
    if (tid == 0) atomicOr(err, 1);
    for (int b = 0; b < 2 && warp != WMMA; ++b) {
      if (!pending[b]) continue;
      uint32_t spins = 0;
      while (!mbar_try(mb[b], phase[b]) && ++spins < kSpinLimit) {
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
  }
  // partial sums: TMEM lane 32 dy + i, column CD (2 - dz) + o of accumulator dx
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp < WMMA && (warp & 3) < 3) {
    const int dy = warp & 3;
    for (int k = warp >> 2; k < 9; k += 2) {
      const int dz = k / 3, dx = k % 3;
      float* out = a.part + (((int64_t)blockIdx.x * 27 + dz * 9 + dy * 3 + dx) * 32 + lane) * CD;
#pragma unroll
      for (int h = 0; h < CD; h += 8) {
        uint32_t v[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(tmem + ((uint32_t)(32 * dy) << 16) + dx * G::N + (2 - dz) * CD + h));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        *reinterpret_cast<uint4*>(out + h) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(out + h + 4) = make_uint4(v[4], v[5], v[6], v[7]);
      }
    }
  }
  float* red = reinterpret_cast<float*>(sm);  // every MMA and copy is done
  if (tid < WWORK)
#pragma unroll
    for (int k = 0; k < 8; ++k) red[tid * 8 + k] = bs[k];
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (tid < CD) {
    float b = 0.f;
    for (int t = tid / 8; t < WWORK; t += G::CH) b += red[t * 8 + tid % 8];
    a.part_b[(int64_t)blockIdx.x * CD + tid] = b;
  }
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(WTMEM));
  }
}

}  // namespace

bool wgrad_tc_ok(int cx, int cd, int nx, int ny) {
  // a plane's offsets are 32-bit
  return cx == 32 && (cd == 32 || cd == 8) && nx % WX == 0 && ny % WY == 0 && (int64_t)nx * ny < (1LL << 26);
}

int wgrad_tc(const WgradArgs& a, int cd, int nsm, int* nblk, cudaStream_t s) {
  const int64_t nsteps = (int64_t)(a.nx / WX) * (a.ny / WY) * a.nlat * a.nz;
  *nblk = (int)std::min<int64_t>(nsteps, nsm);
  auto go = [&](auto kern, int smem) -> int {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return cuda_fail(e, "tcgen05 weight gradient smem attribute");
    kern<<<*nblk, WTHREADS, smem, s>>>(a, a.err);
    if (g_launch_counter) ++*g_launch_counter;
    e = cudaGetLastError();
    return e == cudaSuccess ? LAT_OK : cuda_fail(e, "tcgen05 weight gradient launch");
  };
  return cd == 32 ? go(wgrad_tc_kernel<32>, WgGeom<32>::SMEM) : go(wgrad_tc_kernel<8>, WgGeom<8>::SMEM);
}

}  // namespace net
}  // namespace lat
