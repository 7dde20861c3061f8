// tc05.cuh -- inline-PTX helpers for the 5th-generation tensor cores (tcgen05) on sm_103a:
// tensor-memory allocation, shared-memory matrix descriptors, the single-thread MMA
// issue, commit to an mbarrier with a bounded wait, and tensor-memory loads.
//
// Operand layout used throughout: no swizzle.  A tile of R rows x 64 bf16 is stored as
// core matrices of 8 rows x 16 bytes (128 contiguous bytes, rows 16 bytes apart); core
// matrix (row group g, 16-byte column c) sits at (g * 8 + c) * 128.  The same image
// serves two operands:
//   rows x K (K-major): neighbouring core matrices along K are 128 bytes apart (the
//     descriptor's leading-dimension offset) and neighbouring 8-row groups 1024 bytes
//     apart (its stride-dimension offset).  One kind::f16 MMA consumes K = 16, i.e. two
//     core matrices along K: the k-th MMA of a 64-wide chunk starts 256 * k bytes in.
//   K x columns (MN-major, the row index is K and the 64 columns are M or N): 8-row
//     groups along K are 1024 bytes apart (leading-dimension offset), 8-column groups
//     128 bytes (stride-dimension offset); the k-th MMA starts 2048 * k bytes in.
#pragma once

#include <cstdint>

namespace cgppd {
namespace tc05 {

constexpr int kChunkK = 64;          // bf16 elements per tile row (128 bytes)
constexpr uint32_t kColStep = 128;   // bytes between core matrices adjacent along a row
constexpr uint32_t kRowStep = 1024;  // bytes between 8-row groups

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Byte offset of the 16-byte piece (row r, piece c) of a tile.
__host__ __device__ __forceinline__ uint32_t tile_offset(int r, int c) { return (uint32_t)(((r >> 3) * 8 + c) * 128 + (r & 7) * 16); }

// Shared-memory matrix descriptor: start address, LBO, SBO (all >> 4), descriptor
// version 1 at bits 46-47, base offset 0, absolute LBO mode, no swizzle (bits 61-63 = 0).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Descriptors of a tile as a rows x K operand and as a K x columns operand.
__device__ __forceinline__ uint64_t desc_k_major(uint32_t addr) { return smem_desc(addr, kColStep, kRowStep); }
__device__ __forceinline__ uint64_t desc_mn_major(uint32_t addr) { return smem_desc(addr, kRowStep, kColStep); }

// Instruction descriptor of kind::f16: D f32 (bits 4-5 = 1), A and B bf16 (bits 7-9 and
// 10-12 = 1), A K-major (bit 15 = 0), B K-major or MN-major (bit 16), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N, bool b_mn_major)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Make this thread's generic-proxy shared-memory writes visible to the tensor cores.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.b32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded wait; returns false if the phase did not complete within `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, long long limit = (1ll << 24))
{
    for (long long i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity))
            return true;
    return false;
}

// Announce `bytes` of bulk copies on `bar` (one arrival).
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) from global to
// shared memory; completes on `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst_smem, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     dst_smem),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Bulk copy from shared to global memory in this thread's current bulk group.
__device__ __forceinline__ void bulk_store(void *dst, uint32_t src_smem, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(src_smem), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}

// Every bulk store of this thread has read its shared memory (and, `done`, is written).
__device__ __forceinline__ void bulk_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_store_wait_done() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem], issued by one thread.
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate ? 1u : 0u)
        : "memory");
}

// Arrive on `bar` once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 lanes x 16 columns of 32-bit data: thread i of the warp gets lane (base + i),
// columns col .. col + 15.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v)
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i)
        v[i] = __uint_as_float(r[i]);
}

}  // namespace tc05
}  // namespace cgppd
