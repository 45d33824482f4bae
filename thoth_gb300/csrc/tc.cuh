// tc.cuh — tcgen05 (5th-generation tensor core) building blocks for sm_103a,
// written as inline PTX: TMEM allocation, shared-memory matrix descriptors,
// the BF16 x BF16 -> FP32 MMA issued by one thread, commit to an mbarrier,
// a bounded mbarrier wait, and TMEM -> register loads.
//
// Operand layout (both A and B "K-major", no swizzle): an R x K bf16 operand is
// stored as 8x8 core matrices of 128 contiguous bytes (8 rows x 16 bytes);
// core matrix (rb, kb) sits at byte (kb * (R / 8) + rb) * 128. So the distance
// between core matrices along K (leading byte offset) is R * 16 bytes and the
// distance between 8-row groups (stride byte offset) is 128 bytes.
// D[m][n] = sum_k A[m][k] * B[n][k] — a linear layer Y = X W^T with X as A and
// W (out x in) as B.
#pragma once

#include <cstdint>
#include <cuda_bf16.h>

namespace thoth {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// byte offset of element (r, k) in an R-row K-major core-matrix tile
__host__ __device__ __forceinline__ uint32_t cm_offset(int r, int k, int R)
{
    return (uint32_t)(((k >> 3) * (R >> 3) + (r >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// shared-memory matrix descriptor, SWIZZLE_NONE, K-major
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);        // bits 0-13: start address >> 4
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;     // bits 16-29: leading byte offset >> 4
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;     // bits 32-45: stride byte offset >> 4
    d |= (uint64_t)1 << 46;                         // bits 46-48: fixed 0b001
    // base offset 0, absolute LBO mode 0, layout type 0 (no swizzle)
    return d;
}

// The same tile read as the transposed operand (MN-major, no swizzle): a core matrix holds 8
// elements along M or N (its contiguous 16 bytes) by 8 along K (its rows). So for a tile of
// cm_offset layout the stride between 8-element groups along M or N is the K-major LBO (R * 16
// bytes) and goes into the SBO field, and the stride between 8-row groups along K is 128 bytes
// and goes into the LBO field. One K = 16 slice starts every 256 bytes.
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t saddr, uint32_t R) { return make_desc(saddr, 128, R * 16); }

// instruction descriptor, kind::f16: D = F32, A = B = BF16; a_mn / b_mn: that operand is MN-major
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, bool a_mn = false, bool b_mn = false)
{
    return (1u << 4)                      // D format: F32
           | (1u << 7)                    // A format: BF16
           | (1u << 10)                   // B format: BF16
           | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16)
           | ((uint32_t)(N >> 3) << 17)   // N / 8
           | ((uint32_t)(M >> 4) << 24);  // M / 16
}

// allocate ncols TMEM columns (power of two >= 32) for this CTA; one full warp calls
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
                 "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}

// D[tmem] (+)= A * B^T for one K = 16 slice; single thread
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// arrive on the mbarrier once all previously issued MMAs of this thread complete
__device__ __forceinline__ void mma_commit(uint64_t* mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
        smem_u32(mbar)));
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count));
}

// bounded wait on phase `parity`; returns false after `limit` polls (the caller
// then records an error instead of spinning forever)
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity, uint32_t limit = 1u << 26)
{
    const uint32_t a = smem_u32(mbar);
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(a), "r"(parity));
        if (done) return true;
    }
    return false;
}

// programmatic dependent launch: the next kernel of the stream may be scheduled; everything of the
// previous one is done and visible. Both do nothing in a kernel launched without the attribute.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;"); }

// generic-proxy smem writes -> visible to the tensor core's async proxy
__device__ __forceinline__ void fence_smem_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// one-dimensional bulk copy global -> shared (16-byte aligned, a multiple of 16 bytes), completing
// on the mbarrier, and the barrier's expected byte count with its one arrival
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* mbar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(mbar))
                 : "memory");
}

__device__ __forceinline__ void mbar_expect(uint64_t* mbar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes) : "memory");
}

// barrier initialisation visible to the async proxy
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// 16 consecutive FP32 columns of this thread's TMEM lane, written
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16])
{
    uint32_t r[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(v[i]);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
                   "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
                 : "memory");
}

// the same load without its wait, and the wait: the loaded words pass through it, so nothing that
// uses them can move ahead of it
__device__ __forceinline__ void tmem_ld16_start(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld16_wait(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 16 consecutive FP32 columns of this thread's TMEM lane (32x32b shape)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

} // namespace tc
} // namespace thoth
