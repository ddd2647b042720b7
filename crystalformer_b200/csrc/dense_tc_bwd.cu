// Backward of the dense part of an encoder layer boundary (training), and the weight gradients.
//
//     head of layer l+1    gx  = g_res + gq' Wq + gk Wk + gv Wv,  gq' = gq / 4 + galpha (x) w_pos    (the widths' pipeline)
//     tail of layer l      gh  = (gx W2) [h > 0],  gy = gx + gh W1,  gattn = gy Wo
//
// One kernel per boundary with the organisation of the forward (dense_tc_core.cuh): a tile of 128 rows goes through the
// same twelve 128-deep products with the weights transposed, in the opposite order.  What the weight gradients need (gx,
// gh, gy, gq') is written on the way.
#include "dense_tc_core.cuh"

namespace cf {
namespace {
using namespace tc5;

// gq' = gq / 4 + galpha w_pos of one row (lane l: columns 4 l .. 4 l + 3, head l / 4), written with galpha in place of gq and
// ga: alpha of the head from the saved query (stored divided by 4), then the slope of its width.  The whole warp calls.
__device__ __forceinline__ float4 query_grad(const DenseBackward &p, const float4 &wp, float4 gq, const float4 &qv, float ga, long long row)
{
    const int lane = threadIdx.x & 31;
    const float lb = lane < 16 ? p.lower_bound : p.lower_bound_hi;
    const float slope = p.gauss_scale * (lane < 16 ? p.a_factor : p.a_factor_hi) * p.elu_beta;
    float al = 4.0f * fmaf(qv.w, wp.w, fmaf(qv.z, wp.z, fmaf(qv.y, wp.y, qv.x * wp.x)));
    al += __shfl_xor_sync(FULL, al, 1);
    al += __shfl_xor_sync(FULL, al, 2);
    const float tt = (al + p.gauss_shift) * p.gauss_scale * (p.elu_beta / (1.0f - lb));
    float galpha = ga * slope * (tt > 0.f ? 1.0f : expf(tt));
    if (p.inverse) {
        const float f = (1.0f - lb) * (tt > 0.f ? tt : expm1f(tt)) + 1.0f;
        galpha = -galpha / (f * f);
    }
    gq.x = fmaf(galpha, wp.x, 0.25f * gq.x); gq.y = fmaf(galpha, wp.y, 0.25f * gq.y);
    gq.z = fmaf(galpha, wp.z, 0.25f * gq.z); gq.w = fmaf(galpha, wp.w, 0.25f * gq.w);
    __syncwarp();  // (the lanes of a head have read ga)
    if (row < p.N) {
        *reinterpret_cast<float4 *>(p.gq + row * 128 + 4 * lane) = gq;
        if ((lane & 3) == 0) p.ga[row * HEADS + (lane >> 2)] = galpha;
    }
    return gq;
}

// Chunk c of the hidden units' gradients, gh = (gx W2) [h > 0], as the operand at `a_off` (wait_free: once the previous
// chunk's has been multiplied).
template <class P>
__device__ __forceinline__ void hidden_grads(const DenseBackward &p, const Shared &s, const P &pl, Phase &ph, uint32_t tmem, int d_col,
                                             int done, int c, long long row_base, const float (&xi)[4], float w2_i, const float (&hs)[4],
                                             int a_off, int ready, bool wait_free)
{
    unsigned live = 0u;  // bit 16 half + i: the unit was active
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half) {
        float h[16];
        load_rows(p.h + 128 * c, p.ff, row_base, p.N, pl, half, h);
#pragma unroll
        for (int i = 0; i < 16; ++i) live |= (h[i] > 0.f ? 1u : 0u) << (16 * half + i);
    }
    ph.wait(s, done);
    fence_after();
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half) {
        float g[16];
        tmem_load_16x32(pl.tmem(tmem, d_col, half), g);
#pragma unroll
        for (int i = 0; i < 16; ++i) g[i] = (live >> (16 * half + i)) & 1u ? g[i] * (xi[2 * half + ((i >> 1) & 1)] * w2_i) : 0.f;
        if (half == 0 && wait_free) ph.wait(s, B_A1_FREE);
        store_operand(s.mem + a_off, pl, half, g, hs[2 * half], hs[2 * half + 1]);
        store_rows(p.gh + 128 * c, p.ff, row_base, p.N, pl, half, g);
    }
    fence_async_smem();
    fence_before();
    mbar_arrive(s.bar(ready));
}

template <int ROWS>
__global__ void __launch_bounds__(BLOCK_THREADS, 1) dense_backward_kernel(const DenseBackward p)
{
    extern __shared__ __align__(1024) unsigned char smem_tc[];
    uint32_t tmem;
    const Shared s = block_begin(smem_tc, tmem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long tiles = (p.N + ROWS - 1) / ROWS;
    const int chunks = p.ff / 128;
    const bool head = p.head != nullptr, tail = p.tail != nullptr;

    if (warp == STREAM_WARP) {
        if (lane == 0) {
            Producer pr;
            for (long long tile = blockIdx.x; tile < tiles && pr.ok; tile += gridDim.x) {
                if (head) pr.stream(s, p.head, 0, 3);
                if (tail) pr.stream(s, p.tail, 3, 1 + 2 * chunks);
            }
            if (!pr.ok) pr.drain(s);
        }
    } else if (warp == ISSUE_WARP) {
        if (lane == 0) {
            Issuer is;
            Phase ph;
            for (long long tile = blockIdx.x; tile < tiles && is.ok; tile += gridDim.x) {
                bool ok = true;
                auto ready = [&](int b) { ok = ph.wait(s, b) && ok; fence_after(); };
                auto product = [&](int d, int a, int done) {
                    if (ok) is.product(s, tmem, d, a);
                    ok = ok && is.ok;
                    if (done >= 0) mma_commit(s.bar(done));
                };
                if (head) {
                    ready(B_A0);                     // gq' and gk
                    product(D0, OFF_A0, B_D0);       // (operand 0 is free again)
                    product(D1, OFF_A1, -1);
                    ready(B_A0);                     // gv
                    product(DX, OFF_A0, B_D0);
                }
                if (tail) {
                    ready(B_A0);
                    product(D0, OFF_A0, B_D0);
                    if (chunks > 1) product(D1, OFF_A0, B_D1);
                    for (int c = 0; c < chunks && ok; ++c) {
                        ready(B_A1);
                        product((c & 1) ? DY : DX, OFF_A1, B_A1_FREE);
                        if (c + 2 < chunks) product((c & 1) ? D1 : D0, OFF_A0, (c & 1) ? B_D1 : B_D0);
                    }
                    ready(B_A0);
                    product(D0, OFF_A0, B_D0);
                }
                is.ok = is.ok && ok;
            }
            if (!is.ok) is.drain(s);
        }
    } else {
        using P = PlaceOf<ROWS>;
        const P pl;
        unsigned char *A0 = s.mem + OFF_A0, *A1 = s.mem + OFF_A1;
        const float wh_i = head ? reinterpret_cast<const float *>(p.head)[0] * GIVEN_BACK : 0.f;
        float w2_i = 0.f, w1_i = 0.f, wo_i = 0.f;
        if (tail) {
            const float *inv = reinterpret_cast<const float *>(p.tail);
            w2_i = inv[3] * GIVEN_BACK; w1_i = inv[3 + 2 * chunks - 1] * GIVEN_BACK; wo_i = inv[3 + 2 * chunks] * GIVEN_BACK;
        }
        Phase ph;
        for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const long long row_base = tile * ROWS;
            epilogue_sync();  // the previous tile's readers are done with the per-row scales
            float x[2][16];   // the thread's 32 gradients: gx, then gy
            float xi[4] = {1.f, 1.f, 1.f, 1.f};
            if (head) {
                // ---- gq' and gk as operands 0 and 1, with one scale per row for the three of them (their products meet in
                //      one sum); warp w takes EACH rows, lane l the columns 4 l .. 4 l + 3 (head l / 4)
                constexpr int EACH = P::EACH, STEP = EACH < 4 ? EACH : 4;
                const float4 wp = *reinterpret_cast<const float4 *>(p.w_pos + 4 * lane);
                float *inv_out = s.row_floats(0);
                const uint32_t lane_at = (lane >> 4) * 16384 + (lane & 1) * 8;
                auto put = [&](unsigned char *buf, int row, const float4 v, float sc) {
                    uint2 h0, h1;
                    split_pair(v.x * sc, v.y * sc, h0.x, h1.x);
                    split_pair(v.z * sc, v.w * sc, h0.y, h1.y);
                    unsigned char *c = buf + lane_at + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4);
                    *reinterpret_cast<uint2 *>(c) = h0;
                    *reinterpret_cast<uint2 *>(c + 32768) = h1;
                };
#pragma unroll
                for (int r0 = 0; r0 < EACH; r0 += STEP) {
                    float4 gq[STEP], gk[STEP];
                    float m[STEP];
#pragma unroll
                    for (int u = 0; u < STEP; ++u) {
                        const long long row = row_base + EACH * warp + r0 + u;
                        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                        float4 qv = zero, gvv = zero;
                        gq[u] = gk[u] = zero;
                        float ga = 0.f;
                        if (row < p.N) {
                            gq[u] = *reinterpret_cast<const float4 *>(p.gq + row * 128 + 4 * lane);
                            qv = *reinterpret_cast<const float4 *>(p.q + row * 128 + 4 * lane);
                            gk[u] = *reinterpret_cast<const float4 *>(p.gk + row * 128 + 4 * lane);
                            gvv = *reinterpret_cast<const float4 *>(p.gv + row * 128 + 4 * lane);
                            ga = p.ga[row * HEADS + (lane >> 2)];
                        }
                        gq[u] = query_grad(p, wp, gq[u], qv, ga, row);
                        const float mq = fmaxf(fmaxf(fabsf(gq[u].x), fabsf(gq[u].y)), fmaxf(fabsf(gq[u].z), fabsf(gq[u].w)));
                        const float mk = fmaxf(fmaxf(fabsf(gk[u].x), fabsf(gk[u].y)), fmaxf(fabsf(gk[u].z), fabsf(gk[u].w)));
                        const float mv = fmaxf(fmaxf(fabsf(gvv.x), fabsf(gvv.y)), fmaxf(fabsf(gvv.z), fabsf(gvv.w)));
                        m[u] = fmaxf(mq, fmaxf(mk, mv));
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                        for (int u = 0; u < STEP; ++u) m[u] = fmaxf(m[u], __shfl_xor_sync(FULL, m[u], o));
#pragma unroll
                    for (int u = 0; u < STEP; ++u) {
                        const int row = P::accumulator_row(EACH * warp + r0 + u);
                        float inv;
                        const float sc = power_of_two(m[u], inv);
                        if (lane == 0) inv_out[row] = inv;
                        put(A0, row, gq[u], sc);
                        put(A1, row, gk[u], sc);
                    }
                }
                fence_async_smem();
                fence_before();
                mbar_arrive(s.bar(B_A0));
#pragma unroll
                for (int half = 0; half < P::HALVES; ++half) load_rows(p.g_res, 128, row_base, p.N, pl, half, x[half]);
                epilogue_sync();
#pragma unroll
                for (int i = 0; i < P::HALVES * P::PAIRS; ++i) xi[i] = inv_out[pl.row0 + 8 * i];
                ph.wait(s, B_D0);  // gq' has been multiplied
#pragma unroll
                for (int u = 0; u < EACH; ++u) {
                    const int of_tile = EACH * warp + u, row = P::accumulator_row(of_tile);
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (row_base + of_tile < p.N) v = *reinterpret_cast<const float4 *>(p.gv + (row_base + of_tile) * 128 + 4 * lane);
                    put(A0, row, v, 1.0f / inv_out[row]);  // (powers of two: exact)
                }
                fence_async_smem();
                fence_before();
                mbar_arrive(s.bar(B_A0));
                ph.wait(s, B_D0);
                fence_after();
#pragma unroll
                for (int half = 0; half < P::HALVES; ++half) {
                    float d[16], e[16];
                    tmem_load_16x32(pl.tmem(tmem, D0, half), d);
                    tmem_load_16x32(pl.tmem(tmem, D1, half), e);
#pragma unroll
                    for (int i = 0; i < 16; ++i) d[i] += e[i];
                    tmem_load_16x32(pl.tmem(tmem, DX, half), e);
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[half][i] = fmaf(d[i] + e[i], xi[2 * half + ((i >> 1) & 1)] * wh_i, x[half][i]);
                    store_rows(p.gx, 128, row_base, p.N, pl, half, x[half]);
                }
            } else {
#pragma unroll
                for (int half = 0; half < P::HALVES; ++half) load_rows(p.gx, 128, row_base, p.N, pl, half, x[half]);
            }
            if (!tail) continue;
            publish_rows(s, pl, x, xi);  // gx (read again from memory behind the chunks, whose sum takes its registers)
#pragma unroll
            for (int half = 0; half < P::HALVES; ++half)
#pragma unroll
                for (int i = 0; i < 16; ++i) x[half][i] = 0.f;
            // ---- hidden units: one scale per row for all chunks, |gh| <= 128 max|gx| max|W2| (see the forward)
            float hs[4], hi[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) hs[i] = power_of_two(137438953472.0f * xi[i] * w2_i, hi[i]);
            for (int c = 0; c < chunks; ++c) {
                hidden_grads(p, s, pl, ph, tmem, (c & 1) ? D1 : D0, (c & 1) ? B_D1 : B_D0, c, row_base, xi, w2_i, hs, OFF_A1, B_A1, c > 0);
                if (c > 0) add_accumulator(pl, tmem, (c & 1) ? DX : DY, x);  // of chunk c - 1, beside chunk c's product
            }
            ph.wait(s, B_A1_FREE);
            add_accumulator(pl, tmem, (chunks & 1) ? DX : DY, x);
#pragma unroll
            for (int half = 0; half < P::HALVES; ++half) {
                float g[16];
                load_rows(p.gx, 128, row_base, p.N, pl, half, g);
#pragma unroll
                for (int i = 0; i < 16; ++i) x[half][i] = fmaf(x[half][i], hi[2 * half + ((i >> 1) & 1)] * w1_i, g[i]);
            }
            publish_rows(s, pl, x, xi);  // gy
#pragma unroll
            for (int half = 0; half < P::HALVES; ++half) store_rows(p.gy, 128, row_base, p.N, pl, half, x[half]);
            ph.wait(s, B_D0);
            fence_after();
#pragma unroll
            for (int half = 0; half < P::HALVES; ++half) {
                float d[16];
                tmem_load_16x32(pl.tmem(tmem, D0, half), d);
#pragma unroll
                for (int i = 0; i < 16; ++i) d[i] *= xi[2 * half + ((i >> 1) & 1)] * wo_i;
                store_rows(p.gattn, 128, row_base, p.N, pl, half, d);
            }
        }
    }
    block_end(s, tmem, p.status);
}

// ---- weight gradients ---------------------------------------------------------------------------------------------------
// A block owns one 128 x 128 gradient block (GradJob) and a share of the atom rows, and contracts 64 rows at a time on the
// tensor cores.  The contraction runs over rows, so rows cannot carry scales of their own; the operands are three bfloat16
// pieces (24 bits, the exponent range of float) and a product the six piece products down to 2^-16 relative.  In memory a
// chunk of rows is already what the transposed (MN-major) operand wants: row n of a panel = 64 features of atom n in 128
// swizzled bytes.  Sixteen warps load and convert, one thread issues; two chunks in flight.
// The tensor pipe drops what does not fit when it adds to an accumulator, always towards zero, so a sum that stays in one
// loses half a unit per instruction: 7e-6 of the gradient after 5,000 rows (a float32 GEMM: 3e-7).  Here an accumulator
// holds one chunk, its small products added first, so that four additions are of full size; the chunks are added in
// registers, rounded to nearest (two accumulators, so that the additions of a chunk lie beside the next one's products).
constexpr int GR_ROWS = 64;                                  // atoms per chunk
constexpr int GR_PIECE = GR_ROWS * 256;                      // bytes of one piece of one operand (two 64-feature panels)
constexpr int GR_BUFFER = 6 * GR_PIECE;                      // g pieces, x pieces
constexpr int GR_MISC = 2 * GR_BUFFER;
constexpr int GR_SMEM = GR_MISC + 64 + 16 * 128 * 4;         // barriers, then the warps' column sums
constexpr int GR_THREADS = 544;                              // 16 loader warps, the issuing warp
enum GradBarrier { G_FULL = 0, G_EMPTY = 2, G_DONE = 4 };

__device__ __forceinline__ void split3(float a, float b, uint32_t (&w)[3])
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
        a -= __low2float(h);
        b -= __high2float(h);
    }
}

__global__ void __launch_bounds__(GR_THREADS, 1) weight_grad_kernel(const GradJobs jobs, int splits, float *partial, unsigned *status)
{
    extern __shared__ __align__(1024) unsigned char smem_tc[];
    const GradJob &job = jobs.j[blockIdx.x];
    const uint32_t base = smem_u32(smem_tc);
    volatile unsigned *gave_up = reinterpret_cast<volatile unsigned *>(smem_tc + GR_MISC + 48);
    auto bar = [&](int b) { return base + GR_MISC + 8u * (uint32_t)b; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(bar(G_FULL), 512); mbar_init(bar(G_FULL + 1), 512);
        mbar_init(bar(G_EMPTY), 1); mbar_init(bar(G_EMPTY + 1), 1);
        mbar_init(bar(G_DONE), 1);
        *gave_up = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 16) tmem_alloc<256>(base + GR_MISC + 56);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem_tc + GR_MISC + 56);
    const long long all = (job.rows + GR_ROWS - 1) / GR_ROWS;  // chunks of the job, and this block's share
    const long long c_lo = all * blockIdx.y / splits, c_hi = all * (blockIdx.y + 1) / splits;
    const PlaceOf<128> pl;
    float acc[2][16];  // the accumulator's chunks so far: thread = 4 rows x 8 columns, as in the chain kernels
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i >> 4][i & 15] = 0.f;
    if (warp == 16) {
        if (lane == 0) {
            constexpr uint32_t IDESC = instr_desc<128, 128, 1, true>();
            uint32_t phase = 0;
            bool ok = true;
            for (long long c = c_lo; c < c_hi && ok; ++c) {
                const int b = (int)((c - c_lo) & 1);
                ok = mbar_wait(bar(G_FULL + b), phase, gave_up);
                if (b) phase ^= 1u;
                fence_after();
                if (!ok) break;
                uint64_t g[3], x[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {  // panels of 64 features lie GR_PIECE / 2 apart, groups of eight rows 1 KB
                    g[i] = smem_desc(base + b * GR_BUFFER + i * GR_PIECE, GR_PIECE / 2, 1024);
                    x[i] = smem_desc(base + b * GR_BUFFER + (3 + i) * GR_PIECE, GR_PIECE / 2, 1024);
                }
                const uint32_t d = tmem + 128u * (uint32_t)b;
#pragma unroll
                for (int ks = 0; ks < GR_ROWS / 16; ++ks) {
                    const uint64_t at = (uint64_t)(ks * 2048 >> 4);
                    mma_f16(d, g[2] + at, x[0] + at, IDESC, ks > 0);
                    mma_f16(d, g[0] + at, x[2] + at, IDESC, true);
                    mma_f16(d, g[1] + at, x[1] + at, IDESC, true);
                }
#pragma unroll
                for (int ks = 0; ks < GR_ROWS / 16; ++ks) {
                    const uint64_t at = (uint64_t)(ks * 2048 >> 4);
                    mma_f16(d, g[1] + at, x[0] + at, IDESC, true);
                    mma_f16(d, g[0] + at, x[1] + at, IDESC, true);
                }
#pragma unroll
                for (int ks = 0; ks < GR_ROWS / 16; ++ks) {
                    const uint64_t at = (uint64_t)(ks * 2048 >> 4);
                    mma_f16(d, g[0] + at, x[0] + at, IDESC, true);
                }
                mma_commit(bar(G_EMPTY + b));
            }
            if (!ok) {  // a wait has run out: the instructions issued so far
                unsigned mine = 0u;
                mma_commit(bar(G_DONE));
                mbar_wait(bar(G_DONE), 0, &mine);
            }
        }
    } else {
        // loader: warp w converts rows 4 w .. 4 w + 3 of either operand, lane l the columns 4 l .. 4 l + 3
        uint32_t phase = 1;
        const uint32_t lane_at = (lane >> 4) * (GR_PIECE / 2) + (lane & 1) * 8;
        const bool with_bias = job.bias != nullptr;
        float4 gv[4], xv[4];
        auto fetch = [&](long long c) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const long long row = c * GR_ROWS + 4 * warp + u;
                gv[u] = xv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < c_hi && row < job.rows) {
                    gv[u] = *reinterpret_cast<const float4 *>(job.g + row * job.ldg + 4 * lane);
                    if (job.x_cols == 128) {
                        xv[u] = *reinterpret_cast<const float4 *>(job.x + row * job.ldx + 4 * lane);
                    } else {  // (the features: any number of columns, rows not aligned)
                        const float *xr = job.x + row * job.ldx + 4 * lane;
                        if (4 * lane < job.x_cols) xv[u].x = xr[0];
                        if (4 * lane + 1 < job.x_cols) xv[u].y = xr[1];
                        if (4 * lane + 2 < job.x_cols) xv[u].z = xr[2];
                        if (4 * lane + 3 < job.x_cols) xv[u].w = xr[3];
                    }
                }
            }
        };
        fetch(c_lo);
        float4 sums = make_float4(0.f, 0.f, 0.f, 0.f), lost = sums;  // column sums of g, and what their roundings dropped
        for (long long c = c_lo; c < c_hi + 2; ++c) {  // (the last two only collect)
            const int b = (int)((c - c_lo) & 1);
            unsigned char *gb = smem_tc + b * GR_BUFFER + lane_at, *xb = gb + 3 * GR_PIECE;
            if (c < c_hi || c >= c_lo + 2) mbar_wait(bar(G_EMPTY + b), phase, gave_up);  // (a failed wait is reported at the end)
            if (b) phase ^= 1u;
            if (c >= c_lo + 2) {  // the products of chunk c - 2 are complete
                fence_after();
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float d[16];
                    tmem_load_16x32(pl.tmem(tmem, 128 * b, half), d);
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[half][i] += d[i];
                }
                fence_before();
            }
            if (c >= c_hi) continue;
            if (with_bias) {
                add_compensated((gv[0].x + gv[1].x) + (gv[2].x + gv[3].x), sums.x, lost.x);
                add_compensated((gv[0].y + gv[1].y) + (gv[2].y + gv[3].y), sums.y, lost.y);
                add_compensated((gv[0].z + gv[1].z) + (gv[2].z + gv[3].z), sums.z, lost.z);
                add_compensated((gv[0].w + gv[1].w) + (gv[2].w + gv[3].w), sums.w, lost.w);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int row = 4 * warp + u;
                const uint32_t at = row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4);
                uint32_t lo[3], hi[3];
                split3(gv[u].x, gv[u].y, lo);
                split3(gv[u].z, gv[u].w, hi);
#pragma unroll
                for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2 *>(gb + i * GR_PIECE + at) = make_uint2(lo[i], hi[i]);
                split3(xv[u].x, xv[u].y, lo);
                split3(xv[u].z, xv[u].w, hi);
#pragma unroll
                for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2 *>(xb + i * GR_PIECE + at) = make_uint2(lo[i], hi[i]);
            }
            fence_async_smem();
            mbar_arrive(bar(G_FULL + b));
            fetch(c + 1);
        }
        float4 *mine = reinterpret_cast<float4 *>(smem_tc + GR_MISC + 64) + warp * 32 + lane;
        *mine = make_float4(sums.x + lost.x, sums.y + lost.y, sums.z + lost.z, sums.w + lost.w);
    }
    __syncthreads();
    if (warp < 16) {
        float *out = partial + ((size_t)blockIdx.x * splits + blockIdx.y) * GRAD_PARTIAL;
#pragma unroll
        for (int half = 0; half < 2; ++half) store_rows(out, 128, 0, 128, pl, half, acc[half]);
        if (job.bias != nullptr && threadIdx.x < 128) {
            const float *col = reinterpret_cast<const float *>(smem_tc + GR_MISC + 64) + threadIdx.x;
            float t[16];
#pragma unroll
            for (int w = 0; w < 16; ++w) t[w] = col[128 * w];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int w = 0; w < o; ++w) t[w] += t[w + o];
            out[128 * 128 + threadIdx.x] = t[0];
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 16) tmem_free<256>(tmem);
    if (threadIdx.x == 0) report_waits(gave_up, status);
}

// The splits of a job added in their order and written where the gradient belongs; 16 blocks per job.
__global__ void __launch_bounds__(256) weight_grad_sum_kernel(const GradJobs jobs, int splits, const float *partial)
{
    const GradJob &job = jobs.j[blockIdx.x];
    const float *in = partial + (size_t)blockIdx.x * splits * GRAD_PARTIAL;
    for (int idx = blockIdx.y * 256 + threadIdx.x; idx < 128 * 128 + (job.bias != nullptr ? 128 : 0); idx += gridDim.y * 256) {
        float t = 0.f;
        for (int sp = 0; sp < splits; ++sp) t += in[(size_t)sp * GRAD_PARTIAL + idx];
        if (idx >= 128 * 128) job.bias[idx - 128 * 128] = t;
        else if ((idx & 127) < job.x_cols) job.out[(size_t)(idx >> 7) * job.ldo + (idx & 127)] = t;
    }
}

// Splits of the rows: as many as make the busiest SM finish first (every block costs its chunks of rows plus about three
// chunks' worth of set-up and write-out)
int grad_splits(int count, long long rows)
{
    const long long chunks = (rows + GR_ROWS - 1) / GR_ROWS, sms = sm_count();
    int best = 1;
    double cost = 1e30;
    for (int sp = 1; sp <= GRAD_MAX_SPLITS; ++sp) {
        const long long waves = ((long long)count * sp + sms - 1) / sms;
        const double c = (double)waves * ((double)((chunks + sp - 1) / sp) + 3.0);
        if (c < cost * 0.999) { cost = c; best = sp; }
    }
    return best;
}

}  // namespace

int launch_dense_backward(const DenseBackward &args, cudaStream_t s)
{
    if (args.N == 0) return CF_OK;
    const int waits = check_waits("dense backward");
    if (waits != CF_OK) return waits;
    DenseBackward p = args;
    p.status = wait_status();
    static thread_local DenseLaunch launch;
    const void *const kernels[3] = {reinterpret_cast<const void *>(dense_backward_kernel<128>), reinterpret_cast<const void *>(dense_backward_kernel<64>),
                                    reinterpret_cast<const void *>(dense_backward_kernel<32>)};
    int rc = launch.configure(kernels, "dense backward");
    if (rc != CF_OK) return rc;
    const int rows = tile_rows(p.N);
    const long long blocks = (p.N + rows - 1) / rows, cap = sm_count();
    auto kernel = rows == 128 ? dense_backward_kernel<128> : rows == 64 ? dense_backward_kernel<64> : dense_backward_kernel<32>;
    kernel<<<(unsigned)(blocks < cap ? blocks : cap), tc5::BLOCK_THREADS, tc5::SMEM_BYTES, s>>>(p);
    return launch_status("dense_backward_kernel");
}

size_t grad_partial_floats(int count, long long rows) { return (size_t)count * grad_splits(count, rows) * GRAD_PARTIAL; }

int launch_weight_grads(const GradJobs &jobs, int count, float *partial, cudaStream_t s)
{
    if (count == 0) return CF_OK;
    const int waits = check_waits("weight gradients");
    if (waits != CF_OK) return waits;
    static thread_local bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured[dev & 63]) {
        if (cudaFuncSetAttribute(weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM) != cudaSuccess) {
            cudaGetLastError();
            return fail(CF_ERR_CUDA, "weight gradients: %d bytes of shared memory not available", GR_SMEM);
        }
        configured[dev & 63] = true;
    }
    const int splits = grad_splits(count, jobs.j[0].rows);
    weight_grad_kernel<<<dim3(count, splits), GR_THREADS, GR_SMEM, s>>>(jobs, splits, partial, wait_status());
    weight_grad_sum_kernel<<<dim3(count, 16), 256, 0, s>>>(jobs, splits, partial);
    return launch_status("weight_grad_kernel");
}

}  // namespace cf
