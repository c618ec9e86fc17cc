// umma.cuh -- thin inline-PTX wrappers for the 5th-generation tensor cores (tcgen05) on
// sm_100/sm_103: tensor-memory allocation, the single-thread MMA issue with shared-memory
// operand descriptors, completion through an mbarrier, and the tensor-memory loads of the
// accumulator.  Used by the mixed-precision Cholesky's trailing update (mixed.cu).
#pragma once
#include <cstdint>

namespace capsgpu {
namespace umma {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, canonical K-major layout without swizzle: core
// matrices of 8 rows x 16 bytes stored contiguously (128 B), lbo = byte distance between
// core matrices adjacent in K, sbo = byte distance between 8-row groups; bits 46-47 carry
// the descriptor version (1) of this architecture, bits 61-63 the layout (0: no swizzle)
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) |
           (1ull << 46);
}

// instruction descriptor of kind::tf32: D in FP32, A and B in TF32, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N)
{
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// instruction descriptor of kind::f16 with FP16 A and B: D in FP32, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N)
{
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// one warp, all lanes: ncols columns of tensor memory (power of two >= 32); the base
// address lands in *slot (shared memory)
__device__ __forceinline__ void alloc(uint32_t *slot, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy writes to shared memory become visible to the tensor cores' reads
__device__ __forceinline__ void fence_smem_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// D (+)= A B^T, one thread
__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
// D (+)= A B^T with 16-bit A and B (K = 16 per instruction), one thread
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
// the two words of a K-major descriptor: the low one holds the address (16-byte units) and lbo, so that
// a byte offset o moves it by o / 16; the high one (sbo, version) stays the same.  A single thread
// issues all MMAs of a CTA, and forming 64-bit descriptors in a loop took it longer (150 clocks per
// MMA) than the tensor cores take for a 128 x 64 x 16 one (51; 128 x 128 x 16: 66)
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr, uint32_t lbo) { return (saddr >> 4) | (lbo >> 4) << 16; }
__host__ __device__ constexpr uint32_t desc_hi(uint32_t sbo) { return (sbo >> 4) | 1u << 14; }
template <uint32_t ACC>
__device__ __forceinline__ void mma_f16_lo(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t idesc)
{
    asm volatile("{\n\t.reg .b64 a, b;\n\t.reg .pred p;\n\tmov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}" ::"r"(tmem_d),
                 "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "n"(ACC));
}
// arrive on the mbarrier once every MMA issued so far by this thread has completed
__device__ __forceinline__ void commit(uint64_t *mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t *mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// bounded wait for phase `parity` of the mbarrier; false if it did not complete
__device__ __forceinline__ bool mbar_wait(uint64_t *mbar, uint32_t parity, int max_iter)
{
    uint32_t done = 0;
    for (int it = 0; it < max_iter && !done; it++)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(smem_u32(mbar)), "r"(parity), "r"(10000)
                     : "memory");
    return done != 0;
}

// arrive on the mbarrier and add `bytes` to the transaction count its phase waits for
__device__ __forceinline__ void mbar_arrive_tx(uint64_t *mbar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes) : "memory");
}
// asynchronous bulk copy global -> shared memory of this CTA; completion counts `bytes` off
// the mbarrier's transaction count.  Both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *mbar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"((uint64_t)__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(mbar))
                 : "memory");
}

// 16 consecutive FP32 columns of this warp's 32 lanes (lane = thread)
__device__ __forceinline__ void ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

} // namespace umma
} // namespace capsgpu
