// Fifth-generation tensor core plumbing (sm_100a): mbarriers, bulk copies, tensor memory, tcgen05.mma descriptors, and the
// two-piece half-precision operands of the dense kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cf {
namespace tc5 {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarriers ------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Every wait is bounded: after two seconds (or once another thread of the block has given up) it returns false; the
// caller then leaves its loop, and the block drains its copies, frees its tensor memory and returns.
constexpr unsigned long long WAIT_NS = 2000000000ull;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile unsigned *gave_up, unsigned long long limit_ns = WAIT_NS)
{
    auto ready = [&]() { return mbar_try(bar, parity); };
    if (ready()) return true;
    const unsigned long long t0 = global_ns();
    for (int tries = 0; tries < (1 << 28); ++tries) {
        if (ready()) return true;
        if (*gave_up != 0u) return false;
        if (global_ns() - t0 > limit_ns) break;
    }
    *gave_up = 1u;
    return false;
}

// One thread of a block, at its end: a wait that ran out is reported to the host (wait_status).
__device__ __forceinline__ void report_waits(volatile unsigned *gave_up, unsigned *status)
{
    if (*gave_up != 0u && status != nullptr) atomicOr_system(status, 1u);
}

// ---- copies and proxies ----------------------------------------------------------------------------------------------
// contiguous global -> shared, completion counted in bytes on an mbarrier (addresses and size multiples of 16)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(bar)
                 : "memory");
}
// ordinary shared-memory writes of this thread become visible to tcgen05.mma (the asynchronous proxy)
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- tensor memory ----------------------------------------------------------------------------------------------------
template <int COLUMNS>
__device__ __forceinline__ void tmem_alloc(uint32_t result_smem)  // one whole warp; the address is written to shared memory
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(result_smem), "n"(COLUMNS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int COLUMNS>
__device__ __forceinline__ void tmem_free(uint32_t addr)  // the same warp
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "n"(COLUMNS) : "memory");
}
// 16 lanes x 32 columns of 32-bit accumulators, laid out as the C fragments of four 16 x 8 tiles: register 4 j + u of
// lane (g = lane / 4, t = lane % 4) is row g + 8 (u / 2), column 8 j + 2 t + u % 2.
__device__ __forceinline__ void tmem_load_16x32(uint32_t addr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        " tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");  // (load and wait in one statement: the registers are valid when it ends)
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- matrix instruction -------------------------------------------------------------------------------------------------
// Shared-memory operand descriptor, 128-byte swizzle: rows of 128 bytes, 16-byte chunk c of row r stored at chunk
// c ^ (r & 7).  lbo / sbo in bytes (K-major: sbo = distance of 8-row groups, lbo unused).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::f16, fp32 accumulators, M x N tile; AB = 0: fp16 operands, 1: bf16; MN_MAJOR: both operands transposed
template <int M, int N, int AB, bool MN_MAJOR>
__host__ __device__ constexpr uint32_t instr_desc()
{
    return (1u << 4) | ((uint32_t)AB << 7) | ((uint32_t)AB << 10) | (MN_MAJOR ? (3u << 15) : 0u) | ((uint32_t)(N / 8) << 17) |
           ((uint32_t)(M / 16) << 24);
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
                 : "memory");
}
// the mbarrier is arrived on once all tensor instructions issued so far by this thread have completed
__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- two-piece operands -----------------------------------------------------------------------------------------------
// A value v is stored as h0 + h1, two halves of v s with s a power of two: h0 = half(v s), h1 = half(v s - h0).
// s is chosen so that the largest value of the row (or matrix) that shares it lands in [2^14, 2^15): what is left out is at
// most one unit of v's 24 bits (h0 takes 11, and the rest, which has a sign, needs 12 where h1 has 11: one value in four is
// off, by that unit), with an absolute floor of 2^-25, i.e. 2^-39 of that largest value.  power_of_two gives s and 1 / s for
// a largest magnitude m (exponents clamped so that both are normal numbers; m = 0 is fine).
__device__ __forceinline__ float power_of_two(float m, float &inv)
{
    int e = (int)(__float_as_uint(m) >> 23) & 255;
    e = min(max(e, 16), 254);
    inv = __uint_as_float((uint32_t)(e - 14) << 23);
    return __uint_as_float((uint32_t)(268 - e) << 23);
}
__device__ __forceinline__ void split_pair(float a, float b, uint32_t &h0, uint32_t &h1)
{
    const __half2 hi = __floats2half2_rn(a, b);
    const float2 back = __half22float2(hi);
    const __half2 lo = __floats2half2_rn(a - back.x, b - back.y);
    h0 = *reinterpret_cast<const uint32_t *>(&hi);
    h1 = *reinterpret_cast<const uint32_t *>(&lo);
}
// ... and what is left as a third half: all 24 bits
__device__ __forceinline__ void split_three(float a, float b, uint32_t &h0, uint32_t &h1, uint32_t &h2)
{
    split_pair(a, b, h0, h1);
    const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&h0)), f1 = __half22float2(*reinterpret_cast<const __half2 *>(&h1));
    const __half2 rest = __floats2half2_rn((a - f0.x) - f1.x, (b - f0.y) - f1.y);
    h2 = *reinterpret_cast<const uint32_t *>(&rest);
}

}  // namespace tc5
}  // namespace cf
