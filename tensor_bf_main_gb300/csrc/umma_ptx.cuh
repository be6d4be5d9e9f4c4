// umma_ptx.cuh -- thin inline-PTX wrappers for the sm_100-family (sm_103a)
// asynchronous tensor-core path: mbarriers, TMA tiled loads, the 5th
// generation tensor-core MMA (tcgen05.mma, accumulators in tensor memory)
// and tensor-memory loads.  Every wait here is bounded: after the deadline it
// records where it gave up in a DevStatus word and returns false, so no
// kernel can spin forever.
#pragma once

#include <cuda.h>
#include <stdint.h>

#include "ejoin_internal.cuh"

namespace ejoin {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ----------------------------------------------------------- mbarrier --

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile(
        "{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(
            smem_u32(bar)),
        "r"(bytes)
        : "memory");
}

// Arrive on the barrier at shared::cluster address `addr` (in this CTA or
// another of the cluster, see mapa).  CTA scope: it orders no global-memory
// work of this thread for the other CTA (with cluster scope every arrival
// waited for the thread's earlier global reductions: joins of 4M x 64, pruned,
// BF16 hi+lo, took 24.2 instead of 20.2 ms).  What it hands over here
// is tensor memory whose loads have completed (tcgen05.wait::ld).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

// shared::cluster address of this CTA's shared variable p in CTA `rank`.
__device__ __forceinline__ uint32_t mapa(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// True in one lane of a converged warp (the lane the hardware elects).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(p));
    return p != 0;
}

// All threads of all CTAs of the cluster.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// The hint lets the thread sleep in the instruction for up to 20 us instead of
// returning after a few tens of cycles.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}

// Whether that phase has completed, without waiting.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase of `parity` to complete; false if the deadline passed or
// another role of the kernel already gave up (st->timeout set).
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, DevStatus* st,
                                          unsigned where) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer();
    const uint64_t lim = st->wait_ns ? st->wait_ns : kWaitLimitNs;
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 15u) == 0) {
            if (*(volatile unsigned*)&st->timeout) return false;
            if (globaltimer() - t0 > lim) {
                if (atomicCAS(&st->timeout, 0u, 1u) == 0u) st->where = where;
                return false;
            }
        }
    }
}

// Drain wait before exit: ends when the phase completes or after the same
// deadline, whatever the other roles did (so that no copy or MMA the caller
// issued is left in flight when the CTA exits, unless the hardware stalls).
__device__ __forceinline__ bool mbar_wait_drain(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 15u) == 0 && globaltimer() - t0 > kWaitLimitNs) return false;
    }
}

// Pause of `ns` nanoseconds (bounded by the timer).
__device__ __forceinline__ void pause_ns(uint64_t ns) {
    const uint64_t t0 = globaltimer();
    while (globaltimer() - t0 < ns) __nanosleep(1000);
}

// ---------------------------------------------------------------- TMA --

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// 2-D tiled load of box {x..x+bx, y..y+by} into smem, completing on `bar`.
// x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int32_t x,
                                            int32_t y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(smem_dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// The same load in a CTA pair, completing on the barrier at shared::cluster
// address `bar`, which may lie in the pair's other CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int32_t x,
                                                 int32_t y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(smem_dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// ------------------------------------------------------------ tcgen05 --
//
// CG = 1: one CTA; CG = 2: a pair of CTAs (cluster ranks 0 and 1) that share an
// MMA.  Allocation and release then run in both CTAs, the MMAs and commits in
// rank 0; a commit arrives on the barrier at the same place in both.

// Allocate `ncols` tensor-memory columns (power of two >= 32); the address is
// written to *dst (shared memory).  Whole warp.
template <int CG = 1>
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    if (CG == 2)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(dst)),
                     "r"(ncols)
                     : "memory");
    else
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(dst)),
                     "r"(ncols)
                     : "memory");
}
template <int CG = 1>
__device__ __forceinline__ void tmem_relinquish() {
    if (CG == 2)
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    else
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int CG = 1>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    if (CG == 2)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                     "r"(ncols)
                     : "memory");
    else
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                     "r"(ncols)
                     : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor, K-major operand with the 128-byte swizzle:
// rows of 128 bytes, 8-row (1024-byte) swizzle atoms stacked along M/N.
//   bits  0-13 start address >> 4     bits 16-29 leading byte offset >> 4
//   bits 32-45 stride byte offset >> 4 (1024 B between 8-row groups)
//   bits 46-47 descriptor version (1)  bits 61-63 layout (2 = 128-byte swizzle)
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1u << 46;
    d |= (uint64_t)2u << 61;
    return d;
}

// Same for a K-major operand with the 32-byte swizzle: rows of 32 bytes
// (16 16-bit elements, one K = 16 MMA step), 8-row (256-byte) atoms.
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;
    d |= (uint64_t)(256u >> 4) << 32;
    d |= (uint64_t)1u << 46;
    d |= (uint64_t)6u << 61;
    return d;
}

// Aug operands of packed row p: vals[0..15] the A side, vals[16..31] the B side.
// They are stored as the Gram kernel wants them in shared memory, a 128-row
// tile at a time: 4096 bytes of the A side, then of the B side, rows of 32
// bytes whose 16-byte halves are exchanged in every second group of four rows
// (the 32-byte swizzle).  So a tile is 32 lines of 128 bytes for the copy
// instead of 128 rows of 32 bytes at a pitch of 64, which the copy engine took
// row by row (bare pipeline, 1M x 128 FP16: 95 ms with those rows, 85 ms
// without them).
__device__ __forceinline__ void store_aug(uint16_t* Aug, uint64_t p, const uint16_t (&vals)[32]) {
    const uint32_t r = (uint32_t)p & 127u;
    uint4* t = reinterpret_cast<uint4*>(Aug + (p - r) * 32);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        uint4 w;
        w.x = vals[8 * v + 0] | ((uint32_t)vals[8 * v + 1] << 16);
        w.y = vals[8 * v + 2] | ((uint32_t)vals[8 * v + 3] << 16);
        w.z = vals[8 * v + 4] | ((uint32_t)vals[8 * v + 5] << 16);
        w.w = vals[8 * v + 6] | ((uint32_t)vals[8 * v + 7] << 16);
        t[(v >> 1) * 256 + r * 2 + ((v & 1) ^ ((r >> 2) & 1u))] = w;
    }
}

// Instruction descriptor, dense kind::f16 / kind::f8f6f4 with FP32 accumulate,
// both operands K-major.  a_fmt/b_fmt: kind::f16 0 = F16, 1 = BF16;
// kind::f8f6f4 0 = E4M3.  Bits: 4-5 D format (1 = F32), 7-9 A format,
// 10-12 B format, 17-22 N >> 3, 24-28 M >> 4.
__host__ __device__ constexpr uint32_t idesc_f32acc(uint32_t a_fmt, uint32_t b_fmt, uint32_t M,
                                                    uint32_t N) {
    return (1u << 4) | (a_fmt << 7) | (b_fmt << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by one thread.  In a pair each CTA
// holds half of A's rows and half of B's (at the same shared-memory offsets)
// and gets the accumulator rows of its half of A.
template <int CG = 1>
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                        uint32_t idesc, uint32_t accumulate) {
    if (CG == 2) {
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
        return;
    }
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int CG = 1>
__device__ __forceinline__ void mma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                        uint32_t idesc, uint32_t accumulate) {
    if (CG == 2) {
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
        return;
    }
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrive on `bar` once all previously issued tcgen05 async ops of this thread
// have completed.
template <int CG = 1>
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    if (CG == 2) {
        asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster"
            ".b64 [%0], %1;" ::"r"(smem_u32(bar)),
            "h"((uint16_t)3)
            : "memory");
        return;
    }
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// 32 lanes x 32 columns of 32-bit accumulators: lane l of the warp receives
// row (lane base + l), columns col..col+31.
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
// The same load, with the maximum of the lane's 32 values (FP32) reduced by
// the load itself (tcgen05.ld.red, sm_103a).
__device__ __forceinline__ void tmem_ld_max_32x32b_x32(uint32_t taddr, uint32_t (&r)[32],
                                                       float& mx) {
    asm volatile(
        "tcgen05.ld.red.sync.aligned.32x32b.x32.max.f32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, %32, [%33];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
          "=f"(mx)
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// The same wait, naming the load's destination registers as read and written
// by it, so that the compiler keeps every use of them after the wait (for a
// load left in flight while other work runs).
__device__ __forceinline__ void tmem_ld_wait_regs(uint32_t (&r)[32], float& mx) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                   "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                   "+r"(r[30]), "+r"(r[31]), "+f"(mx)
                 :
                 : "memory");
}

}  // namespace ptx
}  // namespace ejoin
