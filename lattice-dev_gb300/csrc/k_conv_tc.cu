// k_conv_tc.cu -- the closure's 3x3x3 convolutions with 32 output channels
// (32 -> 32, and 4 padded to 8 -> 32) on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory).
//
// A step: one input plane of 256 sites and their halo rows -- two M tiles of
// 128 sites, an M tile being one 128-site x-row (XW = 128) or two 64-site
// x-rows (XW = 64).  Input plane z adds to output planes z-1, z and z+1: the
// three tap planes' weights are N (96 columns), so a step takes 18 MMAs for an
// M tile instead of the 54 of N = 32, and every output still gets its taps in
// the order (dz, dy, dx).  Output planes take turns in eight TMEM slots; a
// step whose three slots wrap round the ring issues its MMAs in two parts.
// Steps are numbered column by column and each block takes an equal run of
// them, marching through z; a run's first and last two steps per column
// complete no output.
//
// Both operands come from shared memory through matrix descriptors in the
// no-swizzle K-major layout (8-row x 16-byte core matrices):
//   A: the 128 rows of one tap are 128 consecutive x of the halo; the tap's
//      x offset is a 16-byte shift.  XW = 128 stores each halo row as 130
//      consecutive x (core matrices 128 B apart).  XW = 64 stores it in
//      groups of 10 positions per 8 sites (x 8g-1 .. 8g+8, core matrices
//      160 B apart), so that a 16-byte shift stays inside a group and the
//      16 core matrices of two consecutive rows sit at one stride.  Four
//      planes are in a ring, three of them in flight;
//   B: the weights [K16 step][channel chunk][tap plane][out 32][8], staged once.
// Sixteen warps run the epilogue of the output plane that the last step
// completed (tcgen05.ld, bias + GELU, or times GELU' for the backward data
// pass), one issues the MMAs, five issue the copies.
//
// What bounds it: the issue of MMAs by one thread was the limit (70 clocks
// each, 108 a step: per-lane code under `lane == 0` moves every operand to
// uniform registers again).  The MMA warp now runs converged and only the
// instruction itself is predicated on the elected lane.  Four 64^3 lattices,
// 32 -> 32 with z stored: 134 us as it was, 115 with N = 96, 91 with the
// converged warp, 89-93 with copies and epilogue in warps of their own (one
// 64^3 lattice: 38.7 -> 33; 128^3: 234 -> 145, 800 TFLOP/s); 4 -> 32: 69 -> 56.  What
// is left: MMAs alone 58, stores and copies 50 each.
//
// Every wait is bounded: a warp that gives up raises a shared abort flag that
// the whole block reads after its next barrier; the block then sets the error
// word, waits (bounded) for its own MMAs, frees its TMEM and returns.
#include <cuda_bf16.h>
#include <stdint.h>

#include <algorithm>

#include "gelu.cuh"
#include "net.hpp"
#include "tc.cuh"

namespace lat {
namespace net {

namespace {

constexpr int TCR = 2;            // M tiles per step
constexpr int MIN_RUN = 4;        // planes a block takes at least (an item fills its ring with two more)
constexpr int CM_BYTES = 128;     // one core matrix: 8 rows x 16 bytes
constexpr int NSLOT = 4;          // ring of halo planes
constexpr int B_CHUNK = 96 * 16;  // bytes per 8-channel chunk of B's rows: 3 tap planes x 32 outputs
constexpr int OSLOT = 8;          // ring of output planes in TMEM
constexpr int TMEM_COLS = TCR * OSLOT * 32;

// warps 0-15: epilogue; warp 16: MMA issue; warps 17-21: copies
constexpr int EPI_WARPS = 16, MMA_WARP = 16, LOAD_WARP = 17, LOADERS = 160;
constexpr int THREADS = 32 * LOAD_WARP + LOADERS;

// shared-memory geometry for CA input channels (32, or 8 = 4 padded) and
// x-rows of XW sites (128 or 64)
template <int CA, int XW>
struct TcGeom {
  static constexpr int CH = CA / 8;                 // 16-byte channel chunks per site
  static constexpr int RPT = 128 / XW;              // y-rows per M tile
  static constexpr int IR = TCR * RPT;              // y-rows per item
  // CA 8 stages one more halo row: the partner rows of the third tap row
  // (finite data, multiplied by zero weights)
  static constexpr int HY = IR + 2 + (CA == 8 ? 1 : 0);
  static constexpr bool GROUPED = XW < 128;
  static constexpr int POS = GROUPED ? XW / 8 * 10 : XW + 2;     // 16-byte positions per halo row and chunk
  static constexpr int SBO = GROUPED ? 160 : CM_BYTES;           // between core matrices along M
  static constexpr int ROW = GROUPED ? POS * 16 : CH * POS * 16;  // between halo y-rows
  static constexpr int CHK = GROUPED ? HY * POS * 16 : POS * 16;  // between channel chunks (K)
  static constexpr int A_PLANE = HY * CH * POS * 16;
  static constexpr int A_BYTES = NSLOT * A_PLANE;
  // K16 steps per input plane and the 16-byte chunks of B they take: CA 32, two
  // steps for each (dy, dx); CA 8, the pairs (dy 0, dx) + (dy 1, dx) and
  // (dy 2, dx) + a zero chunk
  static constexpr int KS = CA == 8 ? 6 : 18;
  static constexpr int B_STEP = 2 * B_CHUNK, B_BYTES = KS * B_STEP;
  // copies of a halo plane: a loader thread takes places (chunk, position) of a
  // row, or (fewer places than threads) every RSTEP-th row of one place
  static constexpr int PLACES = POS * CH;
  static constexpr int NPL = (PLACES + LOADERS - 1) / LOADERS, RSTEP = PLACES < LOADERS ? LOADERS / PLACES : 1;
  static constexpr int SMEM = B_BYTES + A_BYTES + 64;  // + two mbarriers and the TMEM address
  static_assert(!GROUPED || (XW / 8) * SBO == ROW, "the core matrices of an M tile sit at one stride");
  static_assert(SMEM <= 227 * 1024, "shared memory per block");
};

// instruction descriptor: kind::f16, A and B BF16, D FP32, both K-major, M = 128, N = 32 nb
__device__ __forceinline__ uint32_t idesc(uint32_t nb) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((nb * 32u >> 3) << 17) | ((128u >> 4) << 24);
}

template <int CA, int XW, int EPI, bool STORE_Z>
__global__ void __launch_bounds__(THREADS, 1) conv_tc_kernel(ConvArgs a, int* err) {
  using G = TcGeom<CA, XW>;
  constexpr int CHK = G::CHK, ROW = G::ROW, SBO = G::SBO, A_PLANE = G::A_PLANE;
  constexpr int RPT = G::RPT, IR = G::IR;
  constexpr int B_BYTES = G::B_BYTES, A_BYTES = G::A_BYTES;
  extern __shared__ __align__(1024) unsigned char sm[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + B_BYTES + A_BYTES);  // [2]
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + B_BYTES + A_BYTES + 32);
  volatile int* abort = reinterpret_cast<volatile int*>(sm + B_BYTES + A_BYTES + 48);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t b_s = su32(sm), a_s = su32(sm + B_BYTES);
  const uint32_t mb[2] = {su32(mbar), su32(mbar + 1)};

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(su32(tslot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  if (tid == 0) {
    *abort = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mb[0]));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(mb[1]));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // weights [tap][co][ci] (global) -> [K16 step][chunk][tap plane 2, 1, 0][co][8] (shared)
  for (int i = tid; i < G::KS * 2 * 96; i += THREADS) {
    const int n = i % 32, dz = 2 - i / 32 % 3, chunk = i / 96 % 2, ks = i / 192;
    const uint32_t dst = b_s + ks * G::B_STEP + chunk * B_CHUNK + (i % 96) * 16;
    if constexpr (CA == 32) {
      cp16(dst, a.w + ((int64_t)(dz * 9 + ks / 2) * 32 + n) * 32 + (ks % 2 * 2 + chunk) * 8);
    } else {
      const int tap = dz * 9 + (ks < 3 ? 3 * chunk : 6) + ks % 3;
      if (ks >= 3 && chunk)  // (made visible to the tensor core by the fence of step 0)
        *reinterpret_cast<uint4*>(sm + (dst - b_s)) = make_uint4(0, 0, 0, 0);
      else
        cp16(dst, a.w + ((int64_t)tap * 32 + n) * 8);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);

  // epilogue geometry: warp w -> TMEM lanes 32 (w & 3) (sites) of M tile w >> 3, 16 of
  // its 32 columns (channels).  A lane stores whole 32-byte sectors.
  const int quarter = warp & 3, half = warp >> 2 & 1, mtile = warp >> 3 & 1;
  float2 bias[8];
#pragma unroll
  for (int n = 0; n < 8; ++n)
    bias[n] = (EPI == EPI_GELU && a.bias && warp < EPI_WARPS) ? make_float2(a.bias[16 * half + 2 * n], a.bias[16 * half + 2 * n + 1])
                                                               : make_float2(0.f, 0.f);

  const int tiles_x = a.nx / XW, cols_per = tiles_x * (a.ny / IR);
  const int64_t nsteps = (int64_t)cols_per * a.nlat * a.nz;
  const int64_t Nsite = (int64_t)a.nx * a.ny * a.nz;
  uint32_t phase[2] = {0, 0};
  int pending[2] = {0, 0};  // commits not yet waited for, per TMEM buffer
  bool failed = false;

  const int em = 32 * quarter + lane;  // TMEM lane = row of the M tile
  auto site = [&](int64_t lat_base, int x0, int y0, int z) {
    return lat_base + ((int64_t)z * a.ny + (y0 + mtile * RPT + em / XW)) * a.nx + x0 + em % XW;
  };
  // backward: the layer's stored pre-activations of a step, read while its MMAs run
  uint4 zpre[2];
  auto epilogue = [&](int slot, int64_t s) {
    uint32_t v[16];
    const uint32_t taddr = tmem + ((uint32_t)(32 * quarter) << 16) + (mtile * OSLOT + slot) * 32 + 16 * half;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    __align__(16) __nv_bfloat162 o[8];
    if constexpr (EPI == EPI_GELU) {
      __align__(16) __nv_bfloat162 zz[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 zf = __fadd2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), bias[j]);
        zz[j] = __float22bfloat162_rn(zf);
        o[j] = __float22bfloat162_rn(gelu_t2(zf));
      }
      if constexpr (STORE_Z) {
        uint4* zp = reinterpret_cast<uint4*>(a.zout + s * 32 + 16 * half);
        zp[0] = reinterpret_cast<const uint4*>(zz)[0];
        zp[1] = reinterpret_cast<const uint4*>(zz)[1];
      }
    } else {  // EPI_BWD: times GELU'(z) of the layer's stored pre-activation
      __align__(16) __nv_bfloat162 zz[8];
      reinterpret_cast<uint4*>(zz)[0] = zpre[0];
      reinterpret_cast<uint4*>(zz)[1] = zpre[1];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 g = gelu_t_d2(__bfloat1622float2(zz[j]));
        o[j] = __float22bfloat162_rn(
            __fmul2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), g));
      }
    }
    uint4* op = reinterpret_cast<uint4*>(a.out + s * 32 + 16 * half);
    op[0] = reinterpret_cast<const uint4*>(o)[0];
    op[1] = reinterpret_cast<const uint4*>(o)[1];
  };

  // loader threads: places in a halo row and their offsets in a ring slot
  const int lt = tid - 32 * LOAD_WARP;
  const bool loader = warp >= LOAD_WARP && lt < G::PLACES * G::RSTEP;
  const int row0 = G::RSTEP > 1 ? lt / G::PLACES : 0;
  uint32_t soff[G::NPL];
#pragma unroll
  for (int l = 0; l < G::NPL; ++l) {
    const int i = G::RSTEP > 1 ? lt % G::PLACES : lt + l * LOADERS;
    soff[l] = i % G::CH * CHK + i / G::CH * 16;
  }
  // this block's share of all steps (columns of nz planes, one after the other);
  // a run of planes in one column is an item
  int64_t st = nsteps * blockIdx.x / gridDim.x;
  const int64_t st_end = nsteps * (blockIdx.x + 1) / gridDim.x;
  while (st < st_end && !failed) {
    const int64_t col = st / a.nz;
    const int zA = (int)(st % a.nz);
    const int nzs = (int)min((int64_t)(a.nz - zA), st_end - st);
    st += nzs;
    const int64_t li = col / cols_per;
    const int cr = (int)(col % cols_per);
    const int x0 = cr % tiles_x * XW, y0 = cr / tiles_x * IR;
    const __nv_bfloat16* src = a.in + li * Nsite * CA;
    const int64_t lat_base = li * Nsite;
    int goff[G::NPL];  // of the places in a row of the lattice
#pragma unroll
    for (int l = 0; l < G::NPL; ++l) {
      const int i = G::RSTEP > 1 ? lt % G::PLACES : lt + l * LOADERS, c = i % G::CH, p = i / G::CH;
      // position p of a halo row holds x0 + hx - 1
      int x = x0 + (G::GROUPED ? 8 * (p / 10) + p % 10 : p) - 1;
      x = x < 0 ? x + a.nx : (x >= a.nx ? x - a.nx : x);
      goff[l] = x * CA + c * 8;
    }
    // input plane q holds z = zA - 1 + q, in ring slot q & 3; one group per call
    const int nin = nzs + 2;
    auto load_plane = [&](int q) {
      if (q < nin && loader) {
        int z = zA - 1 + q;
        z = z < 0 ? z + a.nz : (z >= a.nz ? z - a.nz : z);
        const __nv_bfloat16* pl = src + (int64_t)z * a.ny * a.nx * CA;
        const uint32_t base = a_s + (q & 3) * A_PLANE;
#pragma unroll 2
        for (int hy = row0; hy < G::HY; hy += G::RSTEP) {
          int y = y0 + hy - 1;
          y = y < 0 ? y + a.ny : (y >= a.ny ? y - a.ny : y);
          const __nv_bfloat16* row = pl + (int64_t)y * a.nx * CA;
#pragma unroll
          for (int l = 0; l < G::NPL; ++l)
            if (l + 1 < G::NPL || G::RSTEP > 1 || lt + l * LOADERS < G::PLACES)
              cp16(base + hy * ROW + soff[l], row + goff[l]);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    load_plane(0);
    load_plane(1);
    load_plane(2);
#pragma unroll 1
    for (int q = 0; q <= nin; ++q) {
      const int buf = q & 1;
      if (q < nin) {
        // plane q has landed (the two after it may be in flight)
        asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        if (*abort) {  // read after the barrier: every thread sees the same value
          failed = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (warp == MMA_WARP) {
          const uint32_t lead = elect_lane();
          // plane q adds to the output planes lo .. hi (tap planes q - o), which are
          // consecutive TMEM slots but where the ring wraps: N = 32 per output
          // plane.  The first K16 step of output plane q overwrites its slot.
          const int lo = max(0, q - 2), hi = min(q, nzs - 1);
          const int n1 = min(hi - lo + 1, OSLOT - (lo & (OSLOT - 1))), n2 = hi - lo + 1 - n1;
          const uint32_t d1 = tmem + (lo & (OSLOT - 1)) * 32, d2 = tmem;
          const uint32_t b1 = (uint32_t)(lo - (q - 2)) * 512, b2 = b1 + n1 * 512;
          // descriptors are affine in the start address: one base per operand, compile-time
          // offsets for the taps (the start-address field never carries: shared addresses
          // stay below 256 KB).  The M tiles take turns.
          const uint64_t ad0 = mdesc(a_s + (q & 3) * A_PLANE, CA == 32 ? CHK : ROW, SBO);
          const uint64_t bd0 = mdesc(b_s, B_CHUNK, CM_BYTES);
          auto a_off = [&](int ks, int r) {
            const int dx = CA == 32 ? ks / 2 % 3 : ks % 3, dy = CA == 32 ? ks / 6 : ks / 3 * 2;
            return (uint64_t)(((dy + r * RPT) * ROW + dx * 16 + (CA == 32 ? ks % 2 * 2 * CHK : 0)) >> 4);
          };
          auto steps = [&](uint32_t d, uint64_t bd, uint32_t id, int ks0) {
#pragma unroll
            for (int ks = 0; ks < G::KS; ++ks)
              if (ks || !ks0) {
#pragma unroll
                for (int r = 0; r < TCR; ++r)
                  mma_bf16(lead, d + r * OSLOT * 32, ad0 + a_off(ks, r), bd + (uint64_t)(ks * G::B_STEP >> 4), id, 1u);
              }
          };
          if (hi == q)
            for (int o = lo; o <= hi; ++o)
#pragma unroll
              for (int r = 0; r < TCR; ++r)
                mma_bf16(lead, tmem + (r * OSLOT + (o & (OSLOT - 1))) * 32, ad0 + a_off(0, r),
                         bd0 + (uint64_t)((o - (q - 2)) * 512 >> 4), idesc(1), o < q ? 1u : 0u);
          steps(d1, bd0 + (b1 >> 4), idesc(n1), hi == q);
          if (n2 > 0) steps(d2, bd0 + (b2 >> 4), idesc(n2), hi == q);
          asm volatile(
              "{\n .reg .pred e;\n setp.ne.b32 e, %1, 0;\n"
              " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(mb[buf]),
              "r"(lead)
              : "memory");
          __syncwarp();
        }
        pending[buf] = 1;
      }
      if (q == 0) {
        load_plane(3);
        continue;
      }
      const int pb = buf ^ 1, o = q - 3;  // MMA(q - 1) completes output plane o
      if constexpr (EPI == EPI_BWD) {
        if (warp < EPI_WARPS && o >= 0) {
          const uint4* zp = reinterpret_cast<const uint4*>(a.zin + site(lat_base, x0, y0, zA + o) * 32 + 16 * half);
          zpre[0] = zp[0];
          zpre[1] = zp[1];
        }
      }
      // bounded wait, agreed within the warp (tcgen05.ld is warp-collective);
      // the MMA warp goes straight to the barrier
      uint32_t spins = 0;
      int to = 0;
      while (warp != MMA_WARP && !mbar_try(mb[pb], phase[pb])) {
        if (++spins > kSpinLimit) {
          to = 1;
          break;
        }
      }
      if (warp == MMA_WARP) {
        // no TMEM reads, no copies
      } else if (__any_sync(0xffffffffu, to)) {
        if (lane == 0) *abort = 1;
      } else {
        phase[pb] ^= 1u;
        pending[pb] = 0;
        load_plane(q + 3);  // into the slot of plane q - 1, which is read
        if (o >= 0 && warp < EPI_WARPS) {
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          epilogue(o & (OSLOT - 1), site(lat_base, x0, y0, zA + o));
        }
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (*abort) failed = true;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  }
  if (failed) {
    if (tid == 0) atomicOr(err, 1);
    // MMAs of a buffer that was not waited for may still be running (the
    // worker warps track the phases; the MMA warp does not wait)
    for (int b = 0; b < 2 && warp != MMA_WARP; ++b) {
      if (!pending[b]) continue;
      uint32_t spins = 0;
      while (!mbar_try(mb[b], phase[b]) && ++spins < kSpinLimit) {
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

// x-row width of the item layout for an nx-wide lattice (0: no layout fits)
int tc_xw(int nx, int ny) {
  if (nx % 128 == 0 && ny % TcGeom<32, 128>::IR == 0) return 128;
  if (nx % 64 == 0 && ny % TcGeom<32, 64>::IR == 0) return 64;
  return 0;
}

template <int XW>
int conv_tc_go(const ConvArgs& a, int ca, int epi, int nsm, int* err, cudaStream_t s) {
  const bool sz = a.zout != nullptr;
  const int64_t nsteps = (int64_t)(a.nx / XW) * (a.ny / TcGeom<32, XW>::IR) * a.nlat * a.nz;
  auto go = [&](auto kern, int smem) -> int {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return cuda_fail(e, "tcgen05 conv smem attribute");
    // Equal runs over all SMs, or runs of a divisor of nz where that is at most
    // two planes longer: a run that goes from one column to the next fills its
    // pipeline twice, which costs about two steps.
    int64_t run = std::max<int64_t>((nsteps + nsm - 1) / nsm, std::min(MIN_RUN, a.nz));
    int64_t div = run;
    while (div < a.nz && a.nz % div) ++div;
    if (div <= run + 2 && div <= a.nz) run = div;
    const unsigned grid = (unsigned)((nsteps + run - 1) / run);
    kern<<<grid, THREADS, smem, s>>>(a, err);
    if (g_launch_counter) ++*g_launch_counter;
    e = cudaGetLastError();
    return e == cudaSuccess ? LAT_OK : cuda_fail(e, "tcgen05 conv launch");
  };
  if (ca == 8) {
    constexpr int sm8 = TcGeom<8, XW>::SMEM;
    if (epi == EPI_BWD) return go(conv_tc_kernel<8, XW, EPI_BWD, false>, sm8);
    return sz ? go(conv_tc_kernel<8, XW, EPI_GELU, true>, sm8) : go(conv_tc_kernel<8, XW, EPI_GELU, false>, sm8);
  }
  constexpr int sm32 = TcGeom<32, XW>::SMEM;
  if (epi == EPI_GELU)
    return sz ? go(conv_tc_kernel<32, XW, EPI_GELU, true>, sm32) : go(conv_tc_kernel<32, XW, EPI_GELU, false>, sm32);
  return go(conv_tc_kernel<32, XW, EPI_BWD, false>, sm32);
}

}  // namespace

bool conv_tc_ok(int ca, int cb, int epi, int nx, int ny) {
  if (!tc_xw(nx, ny) || cb != 32 || epi == EPI_LINEAR) return false;
  return ca == 32 || ca == 8;
}

int conv_tc(const ConvArgs& a, int ca, int epi, int nsm, int* err, cudaStream_t s) {
  const int xw = tc_xw(a.nx, a.ny);
  if (xw == 128) return conv_tc_go<128>(a, ca, epi, nsm, err, s);
  if (xw == 64) return conv_tc_go<64>(a, ca, epi, nsm, err, s);
  return set_error(LAT_ERR_ARG, "tcgen05 conv: nx % 64");
}

}  // namespace net
}  // namespace lat
