// nn_conv.cuh -- Blackwell primitives of the learned initial guess: tensor
// maps, mbarriers, TMA and bulk copies, tcgen05 MMA/TMEM access.
//
// Operand layouts for tcgen05.mma kind::f16 (BF16 in, FP32 accumulate in TMEM).
// Weights: the no-swizzle K-major core-matrix layout; a core matrix is 8 rows x 16
// bytes (8 BF16 along K) stored contiguously, core matrices adjacent along K are
// LBO bytes apart, along M/N SBO bytes apart.  Activations: a TMA box of {c
// channels, pixels} of an NHWC BF16 tensor with the 2c-byte swizzle (c = 16, 32 or
// 64), read K-major by the convolutions (rows are pixels, K the channels; K
// advances by 32 bytes inside the swizzle) and MN-major by the weight gradients
// (rows are channels, K the pixels).  One box of 2c-byte rows replaced c / 8 boxes
// of 16-byte rows, whose rows the TMA unit took one at a time: it bound the
// convolutions.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace nn {

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(saddr(b)),
                 "r"(bytes)
                 : "memory");
}
// bounded wait on phase `parity`; returns false if the limit was reached
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, long limit = (1l << 22)) {
    uint32_t ok = 0;
    for (long it = 0; it < limit; it++) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(saddr(b)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// 4-D tiled TMA load into this CTA's shared memory, completion on `bar`
__device__ __forceinline__ void tma_load4(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                          uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(saddr(dst)),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(saddr(bar))
        : "memory");
}
// contiguous bulk copy global -> shared (16-byte aligned, size multiple of 16)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     saddr(dst)),
                 "l"((uint64_t)src), "r"(bytes), "r"(saddr(bar))
                 : "memory");
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version; base offset 0, no swizzle
    return d;
}
// the same for operands that TMA stored with a 32, 64 or 128-byte swizzle
// (bytes: that many; K-major: sbo = 8 rows of it, MN-major: see k_wgrad.cu)
__device__ __forceinline__ uint64_t smem_desc_swizzled(uint32_t addr, uint32_t lbo, uint32_t sbo, int bytes) {
    const uint64_t mode = bytes == 128 ? 2 : (bytes == 64 ? 4 : 6);
    return smem_desc(addr, lbo, sbo) | mode << 61;
}
// kind::f16 instruction descriptor: D F32, A/B BF16, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = __uint_as_float(r[j]);
}

}  // namespace nn
