// Thin wrappers of the tensor-core (tcgen05), tensor-memory and mbarrier
// instructions the matrix kernels use.  Operands are K-major without swizzle:
// a core matrix is 8 rows of 16 bytes (128 contiguous bytes), consecutive
// 8-row blocks follow each other (SBO = 128) and consecutive 8-element pieces
// of K are `lbo` bytes apart, so element (row, k) sits at
// (k / 8) * lbo + row * 16 + (k % 8) * 2.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace acu {
namespace umma {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo)
{
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
           (1ull << 46);
}

// f16 x f16 -> f32, A and B K-major
__host__ __device__ constexpr uint32_t instr_desc_f16(int M, int N)
{
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Executed by a whole converged warp, which elects the issuing lane inside: a
// branch around the instruction would make its operands (which live in uniform
// registers) be moved there one by one each time, and that took longer than
// the product itself.
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
// (whole warp) arrives once on the barrier when every MMA the elected lane issued before is done
__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
        : "memory");
}
template <int COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t* dst)   // one whole warp
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)), "n"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLS>
__device__ __forceinline__ void tmem_free(uint32_t t)   // the same warp
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(t), "n"(COLS));
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 8 columns of this warp's 32 lanes (a warp reads lanes 32 (warp % 4) ..), as pairs
__device__ __forceinline__ void tmem_ld8(uint32_t t, float2 (&v)[4])
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(t)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
// The loads issued so far are done.  The values pass through, so that nothing
// that uses them can be moved before the wait.
__device__ __forceinline__ void tmem_ld_wait(float2 (&v)[4], float2 (&x)[4])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[1].x), "+f"(v[1].y), "+f"(v[2].x), "+f"(v[2].y), "+f"(v[3].x),
                   "+f"(v[3].y), "+f"(x[0].x), "+f"(x[0].y), "+f"(x[1].x), "+f"(x[1].y), "+f"(x[2].x), "+f"(x[2].y),
                   "+f"(x[3].x), "+f"(x[3].y)::"memory");
}

__device__ __forceinline__ void tmem_ld_wait(float2 (&v)[4])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[1].x), "+f"(v[1].y), "+f"(v[2].x), "+f"(v[2].y), "+f"(v[3].x),
                   "+f"(v[3].y)::"memory");
}

// the same, 16 columns at a time
__device__ __forceinline__ void tmem_ld16(uint32_t t, float2 (&v)[8])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(t)
        : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
__device__ __forceinline__ void tmem_ld_wait(float2 (&v)[8], float2 (&x)[8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[1].x), "+f"(v[1].y), "+f"(v[2].x), "+f"(v[2].y), "+f"(v[3].x),
                   "+f"(v[3].y), "+f"(v[4].x), "+f"(v[4].y), "+f"(v[5].x), "+f"(v[5].y), "+f"(v[6].x), "+f"(v[6].y),
                   "+f"(v[7].x), "+f"(v[7].y), "+f"(x[0].x), "+f"(x[0].y), "+f"(x[1].x), "+f"(x[1].y), "+f"(x[2].x),
                   "+f"(x[2].y), "+f"(x[3].x), "+f"(x[3].y), "+f"(x[4].x), "+f"(x[4].y), "+f"(x[5].x), "+f"(x[5].y),
                   "+f"(x[6].x), "+f"(x[6].y), "+f"(x[7].x), "+f"(x[7].y)::"memory");
}

// registers a thread of this warpgroup may use from here on
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// ---- mbarriers --------------------------------------------------------------
__device__ __forceinline__ void bar_init(uint64_t* b, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_addr(b)),
                 "r"(bytes)
                 : "memory");
}
// Bounded wait for the phase of the given parity; false when it gave up.
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, int limit = 1 << 22)
{
    const uint32_t a = smem_addr(b);
    for (int i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// whether that phase is over, without waiting
__device__ __forceinline__ bool bar_test(uint64_t* b, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(b)), "r"(parity)
        : "memory");
    return ok;
}
// bar_wait for a converged warp, with one answer for all its lanes.
__device__ __forceinline__ bool bar_wait_warp(uint64_t* b, uint32_t parity)
{
    return __all_sync(0xffffffffu, bar_wait(b, parity));
}

// ---- bulk copies (16-byte aligned, sizes multiples of 16) ---------------------
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(src)),
                 "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// the same, added to what is there (FP32, rounded to nearest; subnormals count as zero)
__device__ __forceinline__ void bulk_add(void* dst, const void* src, uint32_t bytes)
{
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst),
                 "r"(smem_addr(src)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// box of a 3-d tensor map at (c0, c1, c2); c0 times the element size is a multiple of 16 bytes
__device__ __forceinline__ void tensor_load_3d(void* dst, const void* map, int c0, int c1, int c2, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_addr(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_addr(bar))
        : "memory");
}
// an empty group, so that groups stay in step
__device__ __forceinline__ void bulk_store_none() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all but the last PENDING groups have read their source
template <int PENDING>
__device__ __forceinline__ void bulk_store_wait_read()
{
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(PENDING) : "memory");
}
// all but the last PENDING groups are done
template <int PENDING = 0>
__device__ __forceinline__ void bulk_store_wait()
{
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(PENDING) : "memory");
}
// bulk operations on global memory that other threads saw done come before those issued from here on
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
// generic-proxy shared-memory writes become visible to MMAs and bulk copies
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

}  // namespace umma
}  // namespace acu
