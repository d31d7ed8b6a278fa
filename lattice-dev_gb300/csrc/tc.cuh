// tc.cuh -- pieces of the tensor-memory kernels (k_conv_tc.cu, k_wgrad_tc.cu):
// descriptors, the MMA instruction, bounded waits.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace lat {
namespace net {

constexpr uint32_t kSpinLimit = 1u << 20;

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp16(uint32_t saddr, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(saddr), "l"(g) : "memory");
}

// shared-memory matrix descriptor, no swizzle: 8 x 16-byte core matrices.  K-major
// operands: lbo between core matrices along K, sbo along M or N; likewise for
// operands whose M or N runs along the 16 bytes (the major-ness is in the
// instruction descriptor)
__device__ __forceinline__ uint64_t mdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this tensor-core generation
  return d;                // base offset 0, absolute LBO mode 0, layout SWIZZLE_NONE (0)
}

// issued by the lane with `lead` set; the whole warp runs up to it, which keeps
// the operands in uniform registers
__device__ __forceinline__ void mma_bf16(uint32_t lead, uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t id,
                                         uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 e, %5, 0;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(id), "r"(acc), "r"(lead));
}
__device__ __forceinline__ uint32_t elect_lane() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e;
}

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(addr), "r"(phase)
      : "memory");
  return ok != 0;
}

}  // namespace net
}  // namespace lat
