// tc05.cuh -- the few tcgen05 (5th-generation tensor core) and mbarrier
// operations the word filters use, as inline PTX for sm_103a.
//
// The filters multiply 0/1 matrices (and small counts) held as E2M1 values:
// kind::mxf4 takes 4-bit operands with one scale per 32 of them, here 1.0
// everywhere, and accumulates in 32-bit floats: exact for every count the
// filters form (checked against popcounts up to 32,768 ones on both sides).
#pragma once
#include <stdint.h>

namespace gsdr {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: false when `limit` polls ran out or another warp gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit,
                                          const volatile int* quit) {
    for (int it = 0; it < limit; it++) {
        if (mbar_try(bar, parity)) return true;
        if (*quit) return false;
    }
    return false;
}

// The same by a whole warp.  (Every lane polls: one lane polling for the others
// adds its divergence to each hand-over, and took half again as long.)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int limit,
                                               const volatile int* quit) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit, quit)) != 0;
}

// All 512 columns of the SM's tensor memory (one CTA per SM: the kernels that
// use it hold most of the shared memory), by one whole warp.
__device__ __forceinline__ void tmem_alloc_all(uint32_t* dst) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(dst))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free_all(uint32_t base) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(base));
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Shared-memory writes of this thread (its completed cp.async copies too) are
// ordered before the MMAs of whoever observes its next arrival.  (It may also
// wait for the thread's loads in flight: issue loads for later stages behind it.)
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Descriptor of a K-major operand tile in shared memory: rows of 128 bytes,
// 16-byte pieces xor-swizzled by the row's low three bits, eight rows per
// 1,024-byte group (1,024-byte aligned).
// The low half moves with the address; the upper is the same for every tile.
__device__ __forceinline__ uint32_t tc_desc_lo(uint32_t addr) {
    return ((addr & 0x3ffffu) >> 4) | (1u << 16);
}
constexpr uint32_t kTcDescHi = 64u | (1u << 14) | (2u << 29);
constexpr int kTcRowBytes = 128;  // 256 E2M1 values
// D[128][n] += A[128][64] B[n][64]^T, E2M1 x E2M1 -> f32
__device__ __forceinline__ uint32_t tc_idesc_fp4(int n) {
    return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24);
}
// Tensor memory columns: two accumulators of up to 240 columns, then the
// scales (every byte of the 32 columns holds 1.0, so their layout is free).
constexpr int kTcMaxN = 240;
constexpr uint32_t kTcScaleA = 480, kTcScaleB = 496;
// The scales, by four warps (warp % 4 = its quarter of the lanes).
__device__ __forceinline__ void tc_fill_scales(uint32_t tmem, int warp) {
    for (uint32_t c = kTcScaleA; c < 512; c++)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(
                         tmem + ((uint32_t)(warp & 3) << 21) + c),
                     "r"(0x7f7f7f7fu));
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// The four MMAs of one 128-byte-wide stage (one thread).  a and b: tc_desc_lo
// of the stage's operands; first: the sums start from zero.
__device__ __forceinline__ void tc_mma_stage(uint32_t d, uint32_t tmem, uint32_t a, uint32_t b,
                                             uint32_t idesc, bool first) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t acc = first && k == 0 ? 0u : 1u;
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            ".reg .b64 da, db;\n\t"
            "setp.ne.u32 p, %4, 0;\n\t"
            "mov.b64 da, {%1, %7};\n\t"
            "mov.b64 db, {%2, %7};\n\t"
            "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], da, db, %3, "
            "[%5], [%6], p;\n\t"
            "}" ::"r"(d),
            "r"(a + 2 * k), "r"(b + 2 * k), "r"(idesc), "r"(acc), "r"(tmem + kTcScaleA),
            "r"(tmem + kTcScaleB), "r"(kTcDescHi)
            : "memory");
    }
}
// The barrier's phase completes when every MMA issued so far has.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}
// Sixteen accumulator columns of this lane's row (a whole warp; warp % 4 is
// the quarter of the lanes it may read); the values are there after
// tc_load_wait.
__device__ __forceinline__ void tc_load16(uint32_t (&r)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
// Waits for this warp's loads; the values pass through so that no use moves
// ahead of it.
__device__ __forceinline__ void tc_load_wait(uint32_t (&r)[16], float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
// 32 bits as 32 E2M1 values (2.0 where the bit is set), in an order that is
// the same for every row: 4-bit field f of word s takes bit 4 f + 2 - s (bit 4 f
// + 3 for s = 3).  Bit 2 of a field is 2.0, and the two shifts to the left can be
// multiplications, off the ALU pipe.
__device__ __forceinline__ uint4 tc_spread(uint32_t v) {
    return make_uint4(v & 0x44444444u, (v * 2u) & 0x44444444u, (v * 4u) & 0x44444444u,
                      (v >> 1) & 0x44444444u);
}
constexpr float kTcSpreadUnit = 0.25f;  // times a sum of products: the count

}  // namespace gsdr
