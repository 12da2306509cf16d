// mma_f8.cuh -- e4m3 products on the tensor cores (tcgen05, sm_100a): operand
// descriptors, the instruction and the wait for its barrier, for scan_mma.cuh and
// for the measurement of the products' rate in intpeak.cu.
#pragma once

#include <cstdint>

namespace cof {

// shared-memory operand descriptor: K-major, no swizzle, rows 16 bytes apart,
// 8-row groups 128 bytes apart, `lead` bytes between 16-byte pieces.  Its low
// half, to which an offset of 16-byte units may be added; the high half is the
// same for all operands.
__device__ __forceinline__ uint32_t mma_desc(uint32_t saddr, uint32_t lead) {
    return ((saddr >> 4) & 0x3FFF) | ((lead >> 4) << 16);
}
constexpr uint32_t kMmaDescHigh = (128 >> 4) | (1u << 14);

template <bool kAccumulate>
__device__ __forceinline__ void mma_f8(uint32_t tmem, uint32_t a, uint32_t b, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 a, {%1, %4};\n\tmov.b64 b, {%2, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, p;\n\t}"
        ::"r"(tmem), "r"(a), "r"(b), "r"(idesc), "r"(kMmaDescHigh), "n"(kAccumulate ? 1 : 0)
        : "memory");
}

// Waits for the barrier's phase (the whole warp); false when `limit` polls did
// not see it.
__device__ __forceinline__ bool mma_wait(uint32_t mbar, uint32_t parity, uint32_t limit) {
    for (uint32_t n = 0; n < limit; ++n) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (__all_sync(0xFFFFFFFFu, done)) return true;
    }
    return false;
}

// instruction descriptor: D f16, A and B e4m3, both K-major, M = 128
__host__ __device__ constexpr uint32_t mma_f8_desc(uint32_t columns) {
    return ((128u >> 4) << 24) | ((columns >> 3) << 17);
}

// a committed product's arrival on the barrier
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
        : "memory");
}

}  // namespace cof
