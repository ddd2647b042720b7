// Pieces shared by the two backward kernels (per-edge operator and fused attention).
//
// The backward of the radial-basis expansion needs, for every (edge, translation) term and head,
//     c_h(d) = sum_k u_h[k] g_k(d),    g_k(d) = exp(-((k+1) mu0 - d)^2 / (2 (wscale mu0)^2)),
// the upstream gradient u (8 x 64, fixed per edge or per atom) contracted with the basis at distance d.  With lanes
// mapped to terms each lane evaluates the 64 basis values of its own term once (64 ex2) and contracts them with u,
// which is read from shared memory with warp-uniform addresses (broadcast, no bank conflicts); no cross-lane
// reduction is needed per term.
#pragma once
#include "lattice_core.cuh"

namespace cf {

constexpr int U_STRIDE = 64;                  // floats per head row of the u tile

// Adds four bins' values of all heads: the even and the odd bins' sums of a head share a packed accumulator (one issue slot
// for two products).
__device__ __forceinline__ void basis_dot_step(const float *__restrict__ u, float &t, float bin_step, float2 (&c2)[8])
{
    const float t1 = t + bin_step, t2 = t1 + bin_step, t3 = t2 + bin_step;
    const float2 g01 = make_float2(ex2(-t * t), ex2(-t1 * t1)), g23 = make_float2(ex2(-t2 * t2), ex2(-t3 * t3));
    t = t3 + bin_step;
#pragma unroll
    for (int h = 0; h < 8; ++h) {
        const float4 uv = *reinterpret_cast<const float4 *>(u + h * U_STRIDE);
        c2[h] = fma2(make_float2(uv.z, uv.w), g23, fma2(make_float2(uv.x, uv.y), g01, c2[h]));
    }
}

// c[h] = sum_k u[h][k] 2^(-((k+1) step - x)^2); u in shared memory, [8][U_STRIDE].
template <int K>
__device__ __forceinline__ void basis_dot(const float *__restrict__ u, float x, float bin_step, float (&c)[8])
{
    float2 c2[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) c2[h] = make_float2(0.f, 0.f);
    float t = bin_step - x;
#pragma unroll 2
    for (int k = 0; k < K; k += 4) basis_dot_step(u + k, t, bin_step, c2);
#pragma unroll
    for (int h = 0; h < 8; ++h) c[h] = c2[h].x + c2[h].y;
}

// The same for a basis of one bin width (BasisParams::windowed): a value more than 8 bins from the term's centre
// xi = x / step - 1 is below 2^-40, so only the 20 bins k0 .. k0 + 19 are evaluated, k0 the multiple of 4 with
// k0 <= floor(xi) - 8 < k0 + 4 (clamped to the table).  The rows of u are then read at lane-dependent offsets.
__device__ __forceinline__ void basis_dot_window(const float *__restrict__ u, float x, float bin_step, float (&c)[8])
{
    float2 c2[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) c2[h] = make_float2(0.f, 0.f);
    int k0 = (__float2int_rd(__fdividef(x, bin_step)) - 9) & ~3;
    k0 = max(0, min(k0, 44));
    float t = (float)(k0 + 1) * bin_step - x;
#pragma unroll
    for (int k = 0; k < 20; k += 4) basis_dot_step(u + k0 + k, t, bin_step, c2);
#pragma unroll
    for (int h = 0; h < 8; ++h) c[h] = c2[h].x + c2[h].y;
}

}  // namespace cf
