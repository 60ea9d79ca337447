// tcgen05 (UMMA) helpers: shared-memory and instruction descriptors, and the
// bounded mbarrier wait every kernel that uses them takes.
#pragma once
#include <cstdint>

// polls after which a wait gives up (the kernel then sets its error flag)
constexpr long long TC_WAIT_POLLS = 1ll << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// tcgen05 shared-memory matrix descriptor, K-major operand without swizzle:
// 8-row x 16-byte core matrices, lbo = bytes between core matrices adjacent
// in K, sbo = bytes between core matrices adjacent in M/N.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of tcgen05
  return d;                // base offset 0, layout: no swizzle
}

// Instruction descriptor of tcgen05.mma kind::f16: FP16 A and B (K-major),
// FP32 accumulator, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_f16(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase, long long polls) {
  for (long long k = 0; k < polls; ++k) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}
