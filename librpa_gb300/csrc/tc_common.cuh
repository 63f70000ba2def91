// Blackwell (sm_103a) primitives in inline PTX: mbarriers with bounded waits,
// TMA tile loads, tcgen05 TMEM allocation / MMA / commit / loads, and the
// shared-memory and instruction descriptors of tcgen05.mma.kind::f16.
//
// Conventions (PTX ISA, tcgen05):
//  * operand tiles in shared memory are K-major, 64 BF16 (128 bytes) per row,
//    written by TMA with 128-byte swizzle; 8 rows form a 1024-byte swizzle atom,
//    so the descriptor stride between 8-row groups (SBO) is 1024 bytes and the
//    start address advances by 32 bytes per K=16 MMA step inside the atom;
//  * the FP32 accumulator of an M=128 MMA occupies TMEM lanes 0..127, one
//    32-bit column per output column; warp w of a warpgroup may read lanes
//    32*(w%4) .. 32*(w%4)+31.
// Every wait is bounded: on timeout the caller records an error code in a
// device flag and leaves the loop instead of spinning forever.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace gb {
namespace tc {

constexpr uint32_t kSpinLimit = 1u << 30;           // polling iterations before a wait is declared failed
constexpr uint64_t kWaitLimitNs = 4000000000ull;    // or 4 s of wall time, whichever comes first

__device__ __forceinline__ uint64_t globaltimer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait; returns false on timeout (iteration count or wall time).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t i = 0; i < kSpinLimit; ++i)
    {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 0 && globaltimer_ns() - t0 > kWaitLimitNs) return false;
    }
    return false;
}

// The same for a wait that is long beside the work of the other warps on its scheduler: it sleeps NAP
// nanoseconds between polls and reads the clock, which costs more than a short wait, every 256 of them.
template <uint32_t NAP>
__device__ __forceinline__ bool mbar_wait_nap(uint64_t *bar, uint32_t parity, uint32_t limit_ms = kWaitLimitNs / 1000000)
{
    uint32_t end = 0;  // of the wait, in units of 2^20 ns (1.05 ms)
    do
    {
#pragma unroll 1
        for (uint32_t i = 0; i < 256; ++i)
        {
            if (mbar_try_wait(bar, parity)) return true;
            if (NAP > 0) __nanosleep(NAP);
        }
        const uint32_t now = static_cast<uint32_t>(globaltimer_ns() >> 20);
        if (end == 0) end = now + limit_ms;
        if (static_cast<int32_t>(now - end) > 0) return false;
    } while (true);
}

// Programmatic dependent launch.  The dependent grid may start once every CTA of this one has called
// pdl_trigger or left; in the dependent, pdl_wait returns when the grids before it are complete and their
// writes visible.  Without the launch attribute both do nothing.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// One lane of a converged warp.  Code that a whole warp runs with this around the issuing instructions
// keeps their operands in uniform registers; under `lane == 0` each operand is moved there first.
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Two FP32 values to BF16, to nearest even, packed (a in the low half)
__device__ __forceinline__ uint32_t bf16x2_rn(float a, float b)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}

// Three-piece BF16 split of a pair of FP32 values, each piece packed as bf16x2 (element 0 in the low half):
// hi and mid to nearest, and lo, which holds what is left exactly: the three together are the value.  To
// nearest, because the products leave out mid x lo, lo x mid and lo x lo: the rms of these over random
// operands is 0.10 x 2^-24 of the product (hi alone to nearest: 0.15, pieces cut off: 0.30).  A call of 16
// atoms of 13/40 on 3x3x3 k: 493 ms with the conversion instructions, 507 with integer additions before a
// cut, 489 with pieces cut off.
__device__ __forceinline__ void split3_pair(float2 e, uint32_t &h, uint32_t &m, uint32_t &l)
{
    constexpr uint32_t top = 0xffff0000u;
    const float2 neg1 = make_float2(-1.0f, -1.0f);
    h = bf16x2_rn(e.x, e.y);
    const float2 r1 = __ffma2_rn(make_float2(__uint_as_float(h << 16), __uint_as_float(h & top)), neg1, e);
    m = bf16x2_rn(r1.x, r1.y);
    const float2 r2 = __ffma2_rn(make_float2(__uint_as_float(m << 16), __uint_as_float(m & top)), neg1, r1);
    l = __byte_perm(__float_as_uint(r2.x), __float_as_uint(r2.y), 0x7632);
}

// 2-D / 3-D TMA tile loads into shared memory, completion counted on an mbarrier.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// L2 cache policy "evict first" (for operands streamed once and not re-read soon).
__device__ __forceinline__ uint64_t l2_policy_evict_first()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// 3-D TMA tile load with an L2 cache policy.
__device__ __forceinline__ void tma_load_3d_hint(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar,
                                                 uint64_t policy)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, "
        "%4}], [%5], %6;" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

// ---- TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t *slot_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D(tmem) (+)= A(smem desc) * B(smem desc)^T, BF16 inputs, FP32 accumulate.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrive on an mbarrier once all previously issued tcgen05.mma of this thread complete.
__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns per warp.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// The same load without the wait: issue several, then tmem_wait_ld() once.
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// 32 lanes x 8 consecutive 32-bit columns per warp, without the wait.
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, SBO = 1024 B, version 1.
__device__ __forceinline__ uint64_t smem_desc_sw128(const void *tile)
{
    const uint64_t addr = smem_u32(tile);
    uint64_t d = 0;
    d |= (addr >> 4) & 0x3FFFull;               // start address
    d |= (uint64_t)(16 >> 4) << 16;             // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;           // stride byte offset between 8-row groups
    d |= 1ull << 46;                            // descriptor version (tcgen05)
    d |= 2ull << 61;                            // SWIZZLE_128B
    return d;
}

// Instruction descriptor: kind::f16, BF16 x BF16 -> FP32, both operands K-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N)
{
    return (1u << 4)                              // D format F32
           | (1u << 7)                            // A format BF16
           | (1u << 10)                           // B format BF16
           | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// Swizzled byte offset inside a [rows][64 bf16] SW128 tile (TMA / tcgen05 canonical layout):
// 16-byte chunk index (0..7) of row r is XOR-ed with (r % 8).
__device__ __forceinline__ uint32_t sw128_offset(int row, int col_bf16)
{
    const int chunk = col_bf16 >> 3;  // 8 bf16 per 16-byte chunk
    const int within = col_bf16 & 7;
    return static_cast<uint32_t>(row * 128 + (((chunk ^ (row & 7)) << 4)) + within * 2);
}

} // namespace tc
} // namespace gb
