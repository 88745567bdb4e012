// Pieces shared by the tcgen05 kernels: shared-memory addresses and descriptors, bounded
// mbarrier waits, tensor maps of BF16 rows.
#pragma once
#include <cuda.h>

#include <cstdint>

#include "pgpu_internal.h"

namespace pgpu {

constexpr uint32_t kTcWaitLimit = 1u << 22;  // polls of a bounded wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// K-major, 128-byte swizzled operand tile (8-row x 128-byte atoms, 1024 bytes apart):
// start address, leading byte offset 16 (unused within one atom), stride byte offset
// 1024, the fixed 0b001 at bits 46-48, swizzle mode 2 (128 B) at bits 61-63.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1u << 16) |
           ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ bool tma_wait(uint32_t bar, uint32_t parity, const volatile int* failed) {
    for (uint32_t it = 0; it < kTcWaitLimit; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.b32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((it & 1023u) == 1023u && *failed) return false;
    }
    return false;
}

__device__ __forceinline__ float gelu_f(float x) {
    return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad_f(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// Tensor maps can be encoded here (the driver offers the call).
bool tensor_maps_available();
// 2-D BF16 tensor map of rows x K values at p, rows rs elements apart (16-byte aligned), box
// 64 (K) x box_rows, 128-byte swizzle, zero fill past the ends.
bool encode_bf16_rows(CUtensorMap* map, const uint16_t* p, uint64_t rows, uint64_t rs, uint32_t K,
                      uint32_t box_rows);

}  // namespace pgpu
