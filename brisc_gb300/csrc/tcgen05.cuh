// tcgen05 (5th-generation tensor core) helpers, inline PTX for sm_103a, shared
// by the restart rotation and the neighbour search.
#pragma once

#include <stdint.h>

#include "tma.cuh"

namespace bgpu {

// Shared-memory matrix descriptor (tcgen05): start address, leading (K) and
// stride (8-row) byte offsets, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo,
                                              uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor, kind::f16: D = F32, A = B = BF16, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t M, uint32_t N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b,
                                         uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accum)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
      ::"r"(smem_u32(bar))
      : "memory");
}

// True in one lane of a converged warp, the one that issues tensor-core work
// (the compiler then needs no loop over lanes around it).
__device__ __forceinline__ bool elect_lane() {
  uint32_t one;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(one));
  return one != 0;
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Bounded wait for phase `parity` of `bar` that gives up when another role has
// raised *stop; a timeout (~2^31 SM cycles) records the error word and
// raises *stop.
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* stop,
                                        int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (*stop) return false;
    if (mbar_try_wait(bar, parity)) return true;
    if (clock64() - t0 > (2LL << 30)) {
      atomicOr(err, kDevErrTimeout);
      *stop = 1;
      return false;
    }
  }
}

}  // namespace bgpu
