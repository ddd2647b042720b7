// Warp-level matrix products on fragments held in registers (mma.sync), and the conversions that feed them.
// Lane (g, t) = (lane / 4, lane % 4).  m16n8k16 (halves): A words (g, 2t), (g + 8, 2t), (g, 2t + 8), (g + 8, 2t + 8); B words
// (2t, g), (2t + 8, g); C (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1).  m16n8k8 (TF32): A (g, t), (g + 8, t), (g, t + 4),
// (g + 8, t + 4); B (t, g), (t + 4, g).
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace cf {

__device__ __forceinline__ void mma_f16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x = hi + lo: hi is x rounded to eleven bits (half away from zero: an integer addition; the conversion instruction is a sequence
// of ten), lo exact.  An infinity or a NaN leaves a NaN in lo.
__device__ __forceinline__ void split_tf32(float x, unsigned &hi, unsigned &lo)
{
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
// Of lo the tensor pipe takes the leading eleven bits; what is left is a third piece.
__device__ __forceinline__ unsigned third_piece(unsigned lo) { return __float_as_uint(__uint_as_float(lo) - __uint_as_float(lo & 0xffffe000u)); }
// What the tensor pipe cuts off a sum is half a unit in its last place on average: MMA_LOST of its value, 2^-24 times the mean of 1 /
// m over mantissas m.
constexpr float MMA_LOST = 4.3e-8f;
// A B + A' B' with three pieces of every operand: as good as float32 sums (two pieces leave 1e-7 of a product).  The large products
// of either half have a sum by themselves, the small ones another together, and what the pipe cuts off is given back.
__device__ __forceinline__ void mma_exact(float (&out)[4], const float (&a)[4], const float (&a2)[4], const unsigned (&bh)[4],
                                          const unsigned (&bl)[4], const unsigned (&b3)[4])
{
    unsigned ah[4], al[4], at[4], ch[4], cl[4], ct[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        split_tf32(a[u], ah[u], al[u]);
        split_tf32(a2[u], ch[u], cl[u]);
        at[u] = third_piece(al[u]);
        ct[u] = third_piece(cl[u]);
    }
    float c[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f}, x[4] = {0.f, 0.f, 0.f, 0.f};
    mma_tf32(x, at, bh[0], bh[1]);
    mma_tf32(x, ct, bh[2], bh[3]);
    mma_tf32(x, ah, b3[0], b3[1]);
    mma_tf32(x, ch, b3[2], b3[3]);
    mma_tf32(x, al, bl[0], bl[1]);
    mma_tf32(x, cl, bl[2], bl[3]);
    mma_tf32(x, al, bh[0], bh[1]);
    mma_tf32(x, cl, bh[2], bh[3]);
    mma_tf32(x, ah, bl[0], bl[1]);
    mma_tf32(x, ch, bl[2], bl[3]);
    mma_tf32(c, ah, bh[0], bh[1]);
    mma_tf32(e, ch, bh[2], bh[3]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const float sum = c[u] + e[u];
        out[u] = sum + fmaf(sum, MMA_LOST, x[u]);
    }
}
__device__ __forceinline__ void split3_tf32(const float (&b)[4], unsigned (&bh)[4], unsigned (&bl)[4], unsigned (&b3)[4])
{
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        split_tf32(b[u], bh[u], bl[u]);
        b3[u] = third_piece(bl[u]);
    }
}
// (x, y) = hi + lo in half pairs
__device__ __forceinline__ void split_f16(float x, float y, unsigned &hi, unsigned &lo)
{
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const unsigned *>(&h);
    lo = *reinterpret_cast<const unsigned *>(&l);
}
// packed pairs of floats, one instruction each
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long &>(d)) : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long &>(d)) : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
    return d;
}
__device__ __forceinline__ float2 half2_of(unsigned w) { return __half22float2(*reinterpret_cast<const __half2 *>(&w)); }
__device__ __forceinline__ unsigned transpose_8x8(unsigned w)
{
    unsigned r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(w));
    return r;
}
__device__ __forceinline__ void ldmatrix4(unsigned (&r)[4], unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(unsigned (&r)[4], unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void copy16_async(unsigned dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

}  // namespace cf
