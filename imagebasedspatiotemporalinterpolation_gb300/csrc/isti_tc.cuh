// Blackwell (sm_103a) primitives for the U-Net kernels, as inline PTX: mbarriers with
// bounded waits, TMA tensor and bulk copies, and the 5th-generation tensor core
// (tcgen05: TMEM allocation, MMA with shared-memory descriptors, commit, TMEM loads).
//
// Operand layout used throughout (the canonical no-swizzle layout of the tcgen05
// shared-memory descriptor): a "core matrix" is 8 rows of 16 contiguous bytes
// (8 bf16 values), 128 bytes in all.  For a K-major operand a row is one M (or N)
// index and its 16 bytes are 8 consecutive K values; the descriptor's leading byte
// offset (LBO) is the distance between core matrices adjacent in K and the stride byte
// offset (SBO) between core matrices adjacent in M/N.  For an MN-major operand a row is
// one K index holding 8 consecutive M (or N) values, and again LBO is the distance
// between core matrices adjacent in K, SBO between those adjacent in M/N.  An NHWC bf16 activation tile
// fetched by TMA as boxes of {8 channels, 16 x, 8 y} lands exactly in this form: 128
// pixels x 16 bytes per box, 8 consecutive pixels per core matrix.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace isti_tc
{
constexpr uint32_t WAIT_LIMIT = 1u << 22; // mbarrier polls before a wait gives up (seconds at most)
constexpr int32_t ERR_TIMEOUT = 4;        // ISTI_ERR_TIMEOUT

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// after the wait for the previous kernel, before TMA reads of what the previous kernel wrote (generic -> async proxy)
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// ---- warp-collective forms ----
//
// The producer and the MMA issuer are whole warps in step: every lane computes the same addresses,
// descriptors and coordinates, and one elected lane executes the copy, MMA or arrival (predicated,
// no branch).  The compiler then keeps those values on the uniform datapath, where the tensor
// instructions take them from; issued from a branch for one lane, each of them moved five or six
// registers over first, at the latency of the move.

// 1 in one lane of the warp (whole warp)
__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n}" : "=r"(e));
    return e;
}

__device__ __forceinline__ void mbar_expect_tx_if(uint32_t leader, uint64_t *bar, uint32_t bytes)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}" ::"r"(smem_u32(bar)),
                 "r"(bytes), "r"(leader)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Waits for the phase with parity `parity` to complete, at most WAIT_LIMIT polls.  On
// timeout the status word is set and false returned: the caller stops its loop.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int32_t *status)
{
    for (uint32_t i = 0; i < WAIT_LIMIT; i++)
        if (mbar_try_wait(bar, parity))
            return true;
    atomicExch(status, ERR_TIMEOUT);
    return false;
}

// mbar_wait by a whole warp in step
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, int32_t *status)
{
    for (uint32_t i = 0; i < WAIT_LIMIT; i++)
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity)))
            return true;
    atomicExch(status, ERR_TIMEOUT);
    return false;
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 4-D tiled TMA load (c, x, y, n) of a tensor map into shared memory (address dst); completion on `bar`.
// c * 2 bytes must be a multiple of 16 (c a multiple of 8 for bf16); x and y may be
// negative or past the end (zero fill).
__device__ __forceinline__ void tma_load_4d(uint32_t leader, uint32_t dst, const CUtensorMap *map, int c, int x, int y, int n, uint64_t *bar)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %7, 0;\n\t"
                 "@p cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n}" ::"r"(dst),
                 "l"(map), "r"(c), "r"(x), "r"(y), "r"(n), "r"(smem_u32(bar)), "r"(leader)
                 : "memory");
}

// 5-D form
__device__ __forceinline__ void tma_load_5d(uint32_t leader, uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t *bar)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %8, 0;\n\t"
                 "@p cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];\n}" ::"r"(
                     dst),
                 "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(bar)), "r"(leader)
                 : "memory");
}

// Untiled bulk copy global -> shared (both 16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load(uint32_t leader, uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n}" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar)), "r"(leader)
                 : "memory");
}

// ---- tcgen05 ----

// Allocates `ncols` TMEM columns (a power of two, 32..512); whole warp.  The address lands
// in shared memory at *dst.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, no swizzle: start address, LBO, SBO (bytes, multiples of
// 16), the fixed version bits 46-48 = 0b001.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: bf16 A and B, f32 accumulator, M x N, operand
// majorness (0 K-major, 1 MN-major).
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t m, uint32_t n, uint32_t a_mn_major, uint32_t b_mn_major)
{
    return (1u << 4)            // D format: f32
           | (1u << 7)          // A format: bf16
           | (1u << 10)         // B format: bf16
           | (a_mn_major << 15) // A major
           | (b_mn_major << 16) // B major
           | ((n >> 3) << 17)   // N >> 3
           | ((m >> 4) << 24);  // M >> 4
}

// A descriptor's low word holds the start address (in units of 16 bytes, below 2^14) and LBO, so
// moving it within shared memory is one 32-bit addition; the high word (SBO, version) stays.  One
// warp issues the MMAs, and what it computes for each of them is what bounds narrow ones
// (N = 32: about 190 cycles an MMA with descriptors built from scratch in a branch for one lane).
struct Desc
{
    uint32_t lo, hi;
    __device__ __forceinline__ Desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
    {
        const uint64_t d = smem_desc(saddr, lbo, sbo);
        lo = (uint32_t)d;
        hi = (uint32_t)(d >> 32);
    }
    // start address + bytes (a multiple of 16)
    __device__ __forceinline__ Desc operator+(uint32_t bytes) const
    {
        Desc d = *this;
        d.lo += bytes >> 4;
        return d;
    }
};

// D[tmem] (+)= A[smem] * B[smem]^T, issued by the elected lane.
__device__ __forceinline__ void mma_bf16(uint32_t leader, uint32_t tmem_d, Desc a, Desc b, uint32_t idesc, bool accumulate)
{
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 q, %7, 0;\n\t"
                 "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}" ::"r"(tmem_d),
                 "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"((uint32_t)accumulate), "r"(leader)
                 : "memory");
}

// Arrives on `bar` once every MMA issued so far by the elected lane has completed.
__device__ __forceinline__ void mma_commit(uint32_t leader, uint64_t *bar)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(smem_u32(bar)), "r"(leader)
                 : "memory");
}

// 32 lanes x 16 columns of 32-bit TMEM words: thread i of the warp gets lane (base lane + i),
// columns col .. col + 15.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
} // namespace isti_tc
