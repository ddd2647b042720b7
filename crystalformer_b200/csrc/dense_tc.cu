// The dense part of an encoder layer boundary in ONE kernel, forward:
//
//     tail of layer l      y  = x + attn Wo^T + bo
//                          x' = y + relu(y W1^T + b1) W2^T + b2            (hidden units in chunks of 128)
//     head of layer l+1    q|k|v = x' Wqkv^T + bqkv ;  a = width(q . w_pos) ;  q <- q / sqrt(16)
//
// (models/indexed_latticeformer_encoder.py:848-890 without LayerNorm, and the in-projection and Gaussian-width
// pipeline of models/indexed_lattice_multi_head_attention_cuda.py:582-722.)  See dense_tc_core.cuh for the organisation
// of a block and the arithmetic.  The chain of a tile alternates products and epilogues; the two products of
// consecutive feed-forward chunks are kept in flight against each other's epilogues (accumulators D0 / D1 for the hidden
// units, DX for the output), so the tensor pipe only waits at y, at x' and at the end of a tile.
#include "dense_tc_core.cuh"

namespace cf {
namespace {
using namespace tc5;

// The rows of attention outputs, element features or species of a tile as operand 0 (scales: row floats 0).
template <class P>
__device__ __forceinline__ void load_first_operand(const DenseForward &p, const Shared &s, long long row_base)
{
    unsigned char *A0 = s.mem + OFF_A0;
    if (p.tail != nullptr) {
        load_operand<P>(s, A0, [&](int row, int ln) {
            return row_base + row < p.N ? *reinterpret_cast<const float4 *>(p.attn + (row_base + row) * 128 + 4 * ln)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
        });
    } else {
        load_operand<P>(s, A0, [&](int row, int ln) {
            float e[4] = {0.f, 0.f, 0.f, 0.f};
            if (row_base + row < p.N) {
                if (p.features != nullptr) {
                    const float *f = p.features + (row_base + row) * p.feature_dim;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (4 * ln + u < p.feature_dim) e[u] = f[4 * ln + u];
                } else {
                    const long long z = p.species[row_base + row] - 4 * ln;
#pragma unroll
                    for (int u = 0; u < 4; ++u) e[u] = z == u ? 1.0f : 0.0f;
                }
            }
            return make_float4(e[0], e[1], e[2], e[3]);
        });
    }
}

// Constants of the weights: 1 / s of each matrix, and a bound of the hidden units' biases (every epilogue thread calls).
struct WeightScales {
    float first = 0.f, w1 = 0.f, w2 = 0.f, head = 0.f, b1_max = 0.f;
    __device__ __forceinline__ WeightScales(const DenseForward &p, const Shared &s)
    {
        const int chunks = p.ff / 128;
        if (p.weights_fresh) grid_dependency_wait();
        if (p.tail != nullptr) {
            const float *inv = reinterpret_cast<const float *>(p.tail);
            first = inv[0] * GIVEN_BACK; w1 = inv[1] * GIVEN_BACK; w2 = inv[2 * chunks] * GIVEN_BACK;
            for (int i = threadIdx.x; i < p.ff; i += EPI_THREADS) b1_max = fmaxf(b1_max, fabsf(p.b1[i]));
            b1_max = warp_max(b1_max);
            if ((threadIdx.x & 31) == 0) s.warp_floats()[threadIdx.x >> 5] = b1_max;
            epilogue_sync();
#pragma unroll
            for (int w = 0; w < EPI_WARPS; ++w) b1_max = fmaxf(b1_max, s.warp_floats()[w]);
        }
        if (p.embed != nullptr) first = *reinterpret_cast<const float *>(p.embed);
        if (p.head != nullptr) head = reinterpret_cast<const float *>(p.head)[1 + 2 * chunks] * GIVEN_BACK;
    }
};

// The thread's 32 features ahead of the feed-forward: x + attn Wo^T + bo, the embedding, or x as it is.
template <class P>
__device__ __forceinline__ void first_rows(const DenseForward &p, const Shared &s, const P &pl, Phase &ph, uint32_t tmem, long long row_base,
                                           float w_i, float (&x)[2][16])
{
    const bool tail = p.tail != nullptr;
    if (!tail && p.embed == nullptr) {
#pragma unroll
        for (int half = 0; half < P::HALVES; ++half) load_rows(p.x_in, 128, row_base, p.N, pl, half, x[half]);
        return;
    }
    load_first_operand<P>(p, s, row_base);
    fence_async_smem();
    fence_before();
    mbar_arrive(s.bar(B_A0));
    float2 bias[4];
    if (tail) {  // the residual and the bias arrive during the product
#pragma unroll
        for (int half = 0; half < P::HALVES; ++half) load_rows(p.x_in, 128, row_base, p.N, pl, half, x[half]);
        load_columns(p.bo, pl, bias);
    }
    epilogue_sync();  // (the loading warps' scales)
    float xi[4];
#pragma unroll
    for (int i = 0; i < P::HALVES * P::PAIRS; ++i) xi[i] = s.row_floats(0)[pl.row0 + 8 * i];
    ph.wait(s, B_D0);
    fence_after();
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half) {
        float d[16];
        tmem_load_16x32(pl.tmem(tmem, D0, half), d);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float sc = xi[2 * half + ((i >> 1) & 1)] * w_i;
            x[half][i] = tail ? x[half][i] + fmaf(d[i], sc, (i & 1) ? bias[i >> 2].y : bias[i >> 2].x) : d[i] * sc;
        }
    }
}

// The hidden units of all chunks share one scale per row (their products with W2 meet in one sum), from a bound known
// beforehand: |h| <= 128 max|y| max|W1| + max|b1|, with both operands below 2^15 in their scaled form.  A bound some 2^8
// above the largest unit still leaves 2^-31 of it as resolution.
__device__ __forceinline__ void hidden_scales(const WeightScales &ws, const float (&xi)[4], float (&hs)[4], float (&hi)[4])
{
#pragma unroll
    for (int i = 0; i < 4; ++i) hs[i] = power_of_two(fmaf(137438953472.0f * xi[i], ws.w1, ws.b1_max), hi[i]);
}

// Chunk c of the hidden units from its accumulator, as the operand at `a_off` (wait_free: once the previous chunk's has
// been multiplied).
template <class P>
__device__ __forceinline__ void hidden_units(const DenseForward &p, const Shared &s, const P &pl, Phase &ph, uint32_t tmem, int d_col,
                                             int done, int c, long long row_base, const float (&xi)[4], float w1_i, const float (&hs)[4],
                                             int a_off, int ready, bool wait_free)
{
    float2 bias[4];
    load_columns(p.b1 + 128 * c, pl, bias);
    ph.wait(s, done);
    fence_after();
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half) {
        float h[16];
        tmem_load_16x32(pl.tmem(tmem, d_col, half), h);
        const float sa = xi[2 * half] * w1_i, sb = xi[2 * half + 1] * w1_i;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 b = bias[j];
            h[4 * j] = fmaxf(fmaf(h[4 * j], sa, b.x), 0.f);
            h[4 * j + 1] = fmaxf(fmaf(h[4 * j + 1], sa, b.y), 0.f);
            h[4 * j + 2] = fmaxf(fmaf(h[4 * j + 2], sb, b.x), 0.f);
            h[4 * j + 3] = fmaxf(fmaf(h[4 * j + 3], sb, b.y), 0.f);
        }
        if (half == 0 && wait_free) ph.wait(s, B_A1_FREE);
        store_operand(s.mem + a_off, pl, half, h, hs[2 * half], hs[2 * half + 1]);
        if (p.h_save != nullptr) store_rows(p.h_save + 128 * c, p.ff, row_base, p.N, pl, half, h);
    }
    fence_async_smem();
    fence_before();
    mbar_arrive(s.bar(ready));
}

// One of q, k, v (which = 0, 1, 2) from its accumulator, and the Gaussian widths beside q.
template <class P>
__device__ __forceinline__ void head_out(const DenseForward &p, const Shared &s, const P &pl, Phase &ph, uint32_t tmem, int d_col,
                                         int done, int which, long long row_base, const float (&xi)[4], float wh_i)
{
    float2 bias[4], w[4];
    load_columns(p.bqkv + 128 * which, pl, bias);
    if (which == 0) load_columns(p.w_pos, pl, w);
    ph.wait(s, done);
    fence_after();
    float *dst = which == 0 ? p.q : which == 1 ? p.k : p.v;
    float al[2][4];  // q . w_pos of the thread's columns: (half, 2 head + row)
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half) {
        float d[16];
        tmem_load_16x32(pl.tmem(tmem, d_col, half), d);
        const float sa = xi[2 * half] * wh_i, sb = xi[2 * half + 1] * wh_i;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 b = bias[j];
            d[4 * j] = fmaf(d[4 * j], sa, b.x); d[4 * j + 1] = fmaf(d[4 * j + 1], sa, b.y);
            d[4 * j + 2] = fmaf(d[4 * j + 2], sb, b.x); d[4 * j + 3] = fmaf(d[4 * j + 3], sb, b.y);
        }
        if (which == 0) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const float2 wa = w[2 * hh], wb = w[2 * hh + 1];
                const float *da = d + 8 * hh, *db = da + 4;
                al[half][2 * hh] = fmaf(db[1], wb.y, fmaf(db[0], wb.x, fmaf(da[1], wa.y, da[0] * wa.x)));
                al[half][2 * hh + 1] = fmaf(db[3], wb.y, fmaf(db[2], wb.x, fmaf(da[3], wa.y, da[2] * wa.x)));
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] *= 0.25f;  // q / sqrt(16)
        }
        store_rows(dst, 128, row_base, p.N, pl, half, d);
    }
    if (which == 0) {
        // the heads' Gaussian widths from alpha = q . w_pos (…attention_cuda.py:647-722): the four lanes of a row trade
        // halves of their sums, lane t finishes head t / 2 of row t % 2 (of either half)
        const float lb = pl.group < 2 ? p.lower_bound : p.lower_bound_hi, factor = pl.group < 2 ? p.a_factor : p.a_factor_hi;
        const float slope = p.gauss_scale * (p.elu_beta / (1.0f - lb));
        const int e = pl.t & 1, hh = pl.t >> 1;
#pragma unroll
        for (int half = 0; half < P::HALVES; ++half) {
            const float *v = al[half];
            const float k0 = (e ? v[1] : v[0]) + __shfl_xor_sync(FULL, e ? v[0] : v[1], 1);
            const float k1 = (e ? v[3] : v[2]) + __shfl_xor_sync(FULL, e ? v[2] : v[3], 1);
            const float alpha = (hh ? k1 : k0) + __shfl_xor_sync(FULL, hh ? k0 : k1, 2);
            const float tt = (alpha + p.gauss_shift) * slope;
            const float elu = tt > 0.f ? tt : expm1f(tt), f = (1.0f - lb) * elu + 1.0f;
            const long long row = row_base + pl.tile0 + 16 * half + 8 * e;
            if (row < p.N && (P::PAIRS == 2 || e == 0)) p.a[row * HEADS + 2 * pl.group + hh] = p.inverse ? factor / f : f * factor;
        }
    }
}

template <int ROWS>
__global__ void __launch_bounds__(BLOCK_THREADS, 1) dense_forward_kernel(const DenseForward p)
{
    extern __shared__ __align__(1024) unsigned char smem_tc[];
    uint32_t tmem;
    const Shared s = block_begin(smem_tc, tmem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long tiles = (p.N + ROWS - 1) / ROWS;
    const int chunks = p.ff / 128;
    const bool tail = p.tail != nullptr, embed = p.embed != nullptr, head = p.head != nullptr;

    if (warp == STREAM_WARP) {
        if (p.weights_fresh) grid_dependency_wait();
        if (lane == 0) {
            Producer pr;
            for (long long tile = blockIdx.x; tile < tiles && pr.ok; tile += gridDim.x) {
                if (tail) pr.stream(s, p.tail, 0, 1 + 2 * chunks);
                else if (embed) pr.stream(s, p.embed, 0, 1, TC_EMBED_PIECES);
                if (head && pr.ok) pr.stream(s, p.head, 1 + 2 * chunks, 3);
            }
            if (!pr.ok) pr.drain(s);
        }
        grid_dependency_wait();
    } else if (warp == ISSUE_WARP) {
        grid_dependency_wait();
        if (lane == 0) {
            Issuer is;
            Phase ph;
            for (long long tile = blockIdx.x; tile < tiles && is.ok; tile += gridDim.x) {
                bool ok = true;
                auto ready = [&](int b) { ok = ph.wait(s, b) && ok; fence_after(); };
                auto product = [&](int d, int a, int done, int pieces = 2) {
                    if (ok) is.product(s, tmem, d, a, pieces);
                    ok = ok && is.ok;
                    mma_commit(s.bar(done));
                };
                if (tail || embed) {
                    ready(B_A0);
                    product(D0, OFF_A0, B_D0, tail ? 2 : TC_EMBED_PIECES);
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
                }
                if (head) {
                    ready(B_A0);
                    product(D0, OFF_A0, B_D0);
                    product(D1, OFF_A0, B_D1);
                    product(DX, OFF_A0, B_DX);
                }
                is.ok = is.ok && ok;
            }
            if (!is.ok) is.drain(s);
        }
    } else {
        using P = PlaceOf<ROWS>;
        const P pl;
        const WeightScales ws(p, s);
        grid_dependency_wait();
        // (not before: the blocks that follow would be packed onto the few SMs that the kernel ahead has left; pooling and head of
        // 128 crystals 30 us behind the last boundary instead of 9)
        grid_launch_dependents();
        Phase ph;
        for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const long long row_base = tile * ROWS;
            epilogue_sync();  // the previous tile's readers are done with the per-row scales
            float x[2][16];   // the thread's 32 features: x, then y, then x'
            float xi[4] = {1.f, 1.f, 1.f, 1.f};  // 1 / scale of its four rows in the current operand
            first_rows(p, s, pl, ph, tmem, row_base, ws.first, x);
            if (tail) {
                publish_rows(s, pl, x, xi);  // y
                // (y lies in memory while the registers take the sum of the chunks, whose hidden units share their scales)
                float *y_rows = p.y_save != nullptr ? p.y_save : p.x_out;
#pragma unroll
                for (int half = 0; half < P::HALVES; ++half) {
                    store_rows(y_rows, 128, row_base, p.N, pl, half, x[half]);
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[half][i] = 0.f;
                }
                float hs[4], hi[4];
                hidden_scales(ws, xi, hs, hi);
                for (int c = 0; c < chunks; ++c) {
                    hidden_units(p, s, pl, ph, tmem, (c & 1) ? D1 : D0, (c & 1) ? B_D1 : B_D0, c, row_base, xi, ws.w1, hs, OFF_A1, B_A1, c > 0);
                    if (c > 0) add_accumulator(pl, tmem, (c & 1) ? DX : DY, x);  // of chunk c - 1, beside chunk c's product
                }
                float2 bias[4];
                load_columns(p.b2, pl, bias);
                ph.wait(s, B_A1_FREE);
                add_accumulator(pl, tmem, (chunks & 1) ? DX : DY, x);
#pragma unroll
                for (int half = 0; half < P::HALVES; ++half) {
                    float y[16];
                    load_rows(y_rows, 128, row_base, p.N, pl, half, y);
                    const float sa = hi[2 * half] * ws.w2, sb = hi[2 * half + 1] * ws.w2;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 b = bias[j];
                        x[half][4 * j] = y[4 * j] + fmaf(x[half][4 * j], sa, b.x);
                        x[half][4 * j + 1] = y[4 * j + 1] + fmaf(x[half][4 * j + 1], sa, b.y);
                        x[half][4 * j + 2] = y[4 * j + 2] + fmaf(x[half][4 * j + 2], sb, b.x);
                        x[half][4 * j + 3] = y[4 * j + 3] + fmaf(x[half][4 * j + 3], sb, b.y);
                    }
                }
            }
            if (head) publish_rows(s, pl, x, xi);
            if (tail || embed) {
#pragma unroll
                for (int half = 0; half < P::HALVES; ++half) store_rows(p.x_out, 128, row_base, p.N, pl, half, x[half]);
            }
            if (!head) continue;
#pragma unroll
            for (int which = 0; which < 3; ++which)
                head_out(p, s, pl, ph, tmem, which == 0 ? D0 : which == 1 ? D1 : DX, which == 0 ? B_D0 : which == 1 ? B_D1 : B_DX, which,
                         row_base, xi, ws.head);
        }
    }
    block_end(s, tmem, p.status);
}

// ---- packing -------------------------------------------------------------------------------------------------------
// A block reads the matrices that share its scale (up to 256 KB) for their largest magnitude, then its own 128 x 128 part:
// bound by the latency of those reads (one float per thread and step: 28 us per launch; sixteen in flight: 16 us).
constexpr int PACK_THREADS = 512;
__global__ void __launch_bounds__(PACK_THREADS) dense_pack_kernel(const PackJob job)
{
    const PackBlock &b = job.b[blockIdx.x];
    __shared__ float warp_m[PACK_THREADS / 32];
    const int tid = threadIdx.x;
    float m = 0.f;
#pragma unroll
    for (int gi = 0; gi < 3; ++gi)
        if (b.group[gi] != nullptr) {
            const float *src = b.group[gi];
            int done = 0;
            if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
                const float4 *src4 = reinterpret_cast<const float4 *>(src);
                const int quads = b.group_elems >> 2;
                done = quads << 2;
#pragma unroll 4
                for (int i = tid; i < quads; i += PACK_THREADS) {
                    const float4 v = __ldg(src4 + i);
                    m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                }
            }
            for (int i = done + tid; i < b.group_elems; i += PACK_THREADS) m = fmaxf(m, fabsf(src[i]));
        }
    m = warp_max(m);
    if ((tid & 31) == 0) warp_m[tid >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < PACK_THREADS / 32; ++w) m = fmaxf(m, warp_m[w]);
    float inv;
    const float sc = power_of_two(m, inv);
    if (tid == 0) reinterpret_cast<float *>(b.image)[b.block] = inv;
    unsigned char *out = b.image + TC_HEADER_BYTES + (size_t)b.block * TC_BLOCK_BYTES;
#pragma unroll 2
    for (int idx = tid; idx < 128 * 16; idx += PACK_THREADS) {
        const int n = idx & 127, k0 = (idx >> 7) * 8;  // a 16-byte chunk: eight k of output row n
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k0 + u;
            v[u] = (n < b.rows && k < b.cols) ? (b.trans ? b.src[(size_t)k * b.ld + n] : b.src[(size_t)n * b.ld + k]) * sc : 0.f;
        }
        uint4 h0, h1, h2;
        split_three(v[0], v[1], h0.x, h1.x, h2.x);
        split_three(v[2], v[3], h0.y, h1.y, h2.y);
        split_three(v[4], v[5], h0.z, h1.z, h2.z);
        split_three(v[6], v[7], h0.w, h1.w, h2.w);
        unsigned char *at = out + (k0 >> 6) * (TC_PIECE_BYTES / 2) + n * 128 + ((((k0 & 63) >> 3) ^ (n & 7)) << 4);
        if (b.pieces == 3) {
            *reinterpret_cast<uint4 *>(at) = h2;
            at += TC_PIECE_BYTES;
        }
        *reinterpret_cast<uint4 *>(at) = h1;
        *reinterpret_cast<uint4 *>(at + TC_PIECE_BYTES) = h0;
    }
}

}  // namespace

int launch_dense_forward(const DenseForward &args, cudaStream_t s)
{
    if (args.N == 0) return CF_OK;
    const int waits = check_waits("dense forward");
    if (waits != CF_OK) return waits;
    DenseForward p = args;
    p.status = wait_status();
    if (p.ff <= 0 || p.ff % 128 != 0 || p.ff > TC_MAX_FF)
        return fail(CF_ERR_UNSUPPORTED, "dense forward: ff_dim=%d must be a multiple of 128 up to %d", p.ff, TC_MAX_FF);
    static thread_local DenseLaunch launch;
    const void *const kernels[3] = {reinterpret_cast<const void *>(dense_forward_kernel<128>), reinterpret_cast<const void *>(dense_forward_kernel<64>),
                                    reinterpret_cast<const void *>(dense_forward_kernel<32>)};
    int rc = launch.configure(kernels, "dense forward");
    if (rc != CF_OK) return rc;
    const int rows = tile_rows(p.N);
    const long long blocks = (p.N + rows - 1) / rows, cap = sm_count();
    auto kernel = rows == 128 ? dense_forward_kernel<128> : rows == 64 ? dense_forward_kernel<64> : dense_forward_kernel<32>;
    launch_chained(kernel, dim3((unsigned)(blocks < cap ? blocks : cap)), dim3(tc5::BLOCK_THREADS), tc5::SMEM_BYTES, s, p.chained, p);
    return launch_status("dense_forward_kernel");
}

int launch_pack(const PackJob &job, int count, cudaStream_t s)
{
    if (count == 0) return CF_OK;
    dense_pack_kernel<<<count, PACK_THREADS, 0, s>>>(job);
    return launch_status("dense_pack_kernel");
}

static PackBlock &pack_add(PackJob &job, int &count, unsigned char *image, int block, const float *src, int ld, int trans)
{
    PackBlock &b = job.b[count++];
    b = PackBlock{};
    b.src = src; b.ld = ld; b.trans = (short)trans; b.rows = 128; b.cols = 128; b.block = (short)block; b.pieces = 2; b.image = image;
    return b;
}

void pack_layer_forward(PackJob &job, int &count, unsigned char *image, int ff, const float *Wq, const float *Wk, const float *Wv,
                        const float *Wo, const float *W1, const float *W2)
{
    const int chunks = ff / 128;
    int at = 0;
    auto one = [&](const float *src, int ld, const float *g0, const float *g1, const float *g2, int elems) {
        PackBlock &b = pack_add(job, count, image, at++, src, ld, 0);
        b.group[0] = g0; b.group[1] = g1; b.group[2] = g2; b.group_elems = elems;
    };
    auto w1 = [&](int c) { one(W1 + (size_t)c * 128 * 128, 128, W1, nullptr, nullptr, ff * 128); };
    one(Wo, 128, Wo, nullptr, nullptr, 128 * 128);
    w1(0);
    if (chunks > 1) w1(1);
    for (int c = 0; c < chunks; ++c) {
        one(W2 + (size_t)c * 128, ff, W2, nullptr, nullptr, ff * 128);
        if (c + 2 < chunks) w1(c + 2);
    }
    one(Wq, 128, Wq, Wk, Wv, 128 * 128);
    one(Wk, 128, Wq, Wk, Wv, 128 * 128);
    one(Wv, 128, Wq, Wk, Wv, 128 * 128);
}

void pack_layer_backward(PackJob &job, int &count, unsigned char *image, int ff, const float *Wq, const float *Wk, const float *Wv,
                         const float *Wo, const float *W1, const float *W2)
{
    const int chunks = ff / 128;
    int at = 0;
    auto one = [&](const float *src, int ld, const float *g0, const float *g1, const float *g2, int elems) {
        PackBlock &b = pack_add(job, count, image, at++, src, ld, 1);
        b.group[0] = g0; b.group[1] = g1; b.group[2] = g2; b.group_elems = elems;
    };
    auto w2 = [&](int c) { one(W2 + (size_t)c * 128, ff, W2, nullptr, nullptr, ff * 128); };
    one(Wq, 128, Wq, Wk, Wv, 128 * 128);
    one(Wk, 128, Wq, Wk, Wv, 128 * 128);
    one(Wv, 128, Wq, Wk, Wv, 128 * 128);
    w2(0);
    if (chunks > 1) w2(1);
    for (int c = 0; c < chunks; ++c) {
        one(W1 + (size_t)c * 128 * 128, 128, W1, nullptr, nullptr, ff * 128);
        if (c + 2 < chunks) w2(c + 2);
    }
    one(Wo, 128, Wo, nullptr, nullptr, 128 * 128);
}

void pack_embedding(PackJob &job, int &count, unsigned char *image, const float *W, int feature_dim)
{
    PackBlock &b = pack_add(job, count, image, 0, W, feature_dim, 0);
    b.cols = (short)feature_dim;
    b.pieces = TC_EMBED_PIECES;
    b.group[0] = W;
    b.group_elems = 128 * feature_dim;
}

}  // namespace cf

extern "C" int64_t cf_dense_image_bytes(int64_t ff_dim) { return (int64_t)(ff_dim > 0 ? cf::tc_image_bytes(cf::tc_layer_blocks((int)ff_dim)) : cf::TC_EMBED_BYTES); }

extern "C" int cf_dense_pack_layer(const float *Wq, const float *Wk, const float *Wv, const float *Wo, const float *W1,
                                   const float *W2, int64_t ff_dim, void *image, void *stream)
{
    using namespace cf;
    CF_REQUIRE(Wq && Wk && Wv && Wo && W1 && W2 && image, CF_ERR_INVALID, "cf_dense_pack_layer: null pointer");
    CF_REQUIRE(ff_dim > 0 && ff_dim % 128 == 0 && ff_dim <= TC_MAX_FF, CF_ERR_UNSUPPORTED,
               "cf_dense_pack_layer: ff_dim=%lld must be a multiple of 128 up to %d", (long long)ff_dim, TC_MAX_FF);
    CF_REQUIRE((reinterpret_cast<uintptr_t>(image) & 15) == 0, CF_ERR_INVALID, "cf_dense_pack_layer: image must be 16-byte aligned");
    PackJob job;
    int count = 0;
    pack_layer_forward(job, count, static_cast<unsigned char *>(image), (int)ff_dim, Wq, Wk, Wv, Wo, W1, W2);
    return launch_pack(job, count, as_stream(stream));
}

extern "C" int cf_dense_pack_embedding(const float *W, int64_t feature_dim, void *image, void *stream)
{
    using namespace cf;
    CF_REQUIRE(W && image, CF_ERR_INVALID, "cf_dense_pack_embedding: null pointer");
    CF_REQUIRE(feature_dim >= 1 && feature_dim <= 128, CF_ERR_UNSUPPORTED, "cf_dense_pack_embedding: %lld features (1..128)", (long long)feature_dim);
    CF_REQUIRE((reinterpret_cast<uintptr_t>(image) & 15) == 0, CF_ERR_INVALID, "cf_dense_pack_embedding: image must be 16-byte aligned");
    PackJob job;
    int count = 0;
    pack_embedding(job, count, static_cast<unsigned char *>(image), W, (int)feature_dim);
    return launch_pack(job, count, as_stream(stream));
}
