// Infinitely connected attention over pair grids (pair_grid.cuh), backward: gradients of q, a and, per edge, what those of k and v are
// summed from.  With u_h = W_h^T gout_h, c_h[m] = sum_k u_h[k] g_k(d_m), delta_h = gout_h . out_h, dv_h[j] = gout_h . v_j - delta_h and
// w_h[j] = exp(q.k_j - lse):
//     S0 = sum_m rho x    S1 = sum_m rho x c    S2 = sum_m rho x d^2    S3 = sum_m rho x c d^2        (x = exp(a d^2); heads and keys)
//     p = w S0            glogit = w (S1 + S0 dv)            ga = sum_j w (S2 dv + S3)            gq = sum_j glogit k_j
// which is the chain of infinite_attn_bwd.cu with the images summed in rho: four products of the (keys x nodes) matrix rho with
// eight columns.
//
// Block = eight rows of a crystal.  (1) warp = head: logits, gout.v and u of the eight rows, by products.  (2) warp = row: the four
// products, three node tiles at a time (their columns are 48 registers), every pass over all keys; p and glogit add up in the
// tables.  (3) warp = head: gq.
//
// Bound: issue and latency of a warp's chain (128 registers: 16 warps on an SM; 8 beyond 48 atoms, where the tables of one block
// fill it); the vectors come from L2.  256 crystals of up to 40 atoms: 78 us per layer (112 with 8 warps on an SM, u apart from the
// sums), 169 by term lists (infinite_attn_bwd.cu), whose work grows with the images.  Issue slots 48 %, tensor
// pipe 32 %, LSU wavefronts 38 %.  Error against 64 bits over 40 draws (gq, gk, gv, ga): 2.4, 2.4, 1.0, 3.3e-7, by enumeration 3.9, 3.8,
// 1.1, 4.2e-7; S0's small products add up apart from the large ones (gv 1.04e-7 instead of 1.0 without, small logits).
#include "pair_attn.cuh"

namespace cf {
namespace {

constexpr int PASS = PA_STEP, STAGES = 2;
constexpr int WARPS = PG_ROWS, THREADS = 32 * WARPS;
constexpr int RING = (KeyRing<STAGES>::BYTES + 127) / 128 * 128;
constexpr int U_LD = 512 + 4;

struct Args {
    const float *q, *k, *v, *a, *rvlen, *W, *out, *gout, *lse;
    const int64_t *edge_start;
    BoxRule rule;
    PairGridParams par;
    const unsigned char *slots;
    const int4 *tiles;
    const unsigned *counters;
    const unsigned char *left;
    const uint4 *basis_nodes;
    float inv_wscale;
    float c_scale, c_unit, n2_scale, ga_unit;  // see column_scales
    float *gq, *ga, *glogit, *prob;
    int max_atoms;
};

// logits, gout.v, p and glogit of a row, each in the order of the sums S
__host__ __device__ constexpr int table_words(int max_atoms) { return ((max_atoms + PA_KEYS - 1) / PA_KEYS) * 128 + 4; }
// p and glogit of a row lie side by side, and there its u before
__host__ __device__ constexpr int sums_words(int max_atoms, bool basis)
{
    return basis && 2 * table_words(max_atoms) - 4 < U_LD ? U_LD : 2 * table_words(max_atoms) - 4;
}
size_t smem_bytes(int max_atoms, bool basis)
{
    return (size_t)WARPS * RING + sizeof(float) * PG_ROWS * (2 * table_words(max_atoms) + sums_words(max_atoms, basis));
}

// x f as the operand of a product over the nodes (nodes x heads), f given at nodes g, g + 8 and heads 2t, 2t + 1
__device__ __forceinline__ void node_operand(const float (&f)[4], unsigned (&h)[2], unsigned (&l)[2])
{
    split_f16(f[0], f[1], h[0], l[0]);
    split_f16(f[2], f[3], h[1], l[1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) { h[u] = transpose_8x8(h[u]); l[u] = transpose_8x8(l[u]); }
}

// Powers of two that keep the columns within half precision (65,504) whatever the widths.  x comes as 2^15 at most, u as 2^11, the
// basis as 2^14.
// c = sum_k u_k g_k(d) <= u_max sum_k g_k(d), and sum_k exp(-(y - k)^2 / 2 w^2) <= 1 + sqrt(2 pi) w for any y (the largest term, and the
// integral of the others): x c is at most 2^13 (1 + sqrt(2 pi) w) after 2^-27, which fits up to w = 2.75 and is halved from there on
// as often as it takes.
// x n^2 is at most 2 / e of s^2, s the Gaussian's standard deviation in node spacings; a row's nodes reach down to 2^floor with
// PA_USUAL_LAG bits to spare, so s^2 <= (nodes)^2 / (2 ln 2 (PA_USUAL_LAG - floor)): 420 at the floor of 2^-30, 2^-9 then.  Scaled to 1 at
// most, it leaves x c n^2 below x c.
void column_scales(Args &p, double wscale)
{
    int down = 27;
    for (double most = 8192.0 * (1.0 + 2.5066282746310002 * wscale); most > 65000.0; most *= 0.5) ++down;
    p.c_scale = (float)ldexp(1.0, -down);
    p.c_unit = (float)ldexp(1.0, down);
    const double nodes = p.par.tiles * PG_TILE - PG_POINTS, s2 = nodes * nodes / (2.0 * 0.6931471805599453 * fmax(PA_USUAL_LAG - (double)p.par.floor_log2, 1.0));
    int n2 = 9;
    while (0.7357588823428847 * s2 > ldexp(1.0, n2)) ++n2;
    p.n2_scale = (float)ldexp(1.0, -n2);
    p.ga_unit = (float)ldexp(1.0 / ((double)p.par.inv_h2 + (double)p.par.inv_h2_low), n2);
}

template <bool BASIS>
__global__ void __launch_bounds__(THREADS, 2) pair_attn_bwd_kernel(const Args p)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(FULL, tid >> 5, 0), g = lane >> 2, t = lane & 3;
    const int row_words = table_words(p.max_atoms);
    float *logits = reinterpret_cast<float *>(smem + WARPS * RING), *dvs = logits + PG_ROWS * row_words;
    const int sums_ld = sums_words(p.max_atoms, BASIS);
    float *probs = dvs + PG_ROWS * row_words, *glogits = probs + row_words, *us = probs;
    __shared__ int there[PG_ROWS];
    if (blockIdx.x >= p.counters[0]) return;
    const int4 tile = p.tiles[2 * blockIdx.x], place = p.tiles[2 * blockIdx.x + 1];
    const int i0 = tile.y, n = tile.z, rows = min(PG_ROWS, n - i0);
    if (n < 0 || n > p.max_atoms) return;  // (all its rows are left over)
    const long long a0 = tile.w;
    const int key_tiles = (n + PA_KEYS - 1) / PA_KEYS, i = i0 + min(warp, rows - 1);
    const long long e0 = p.edge_start[tile.x] + (long long)i * n;  // the row's first edge

    const long long my_row = (a0 + min(i0 + g, n - 1)) * (HEADS * HEAD_DIM) + warp * HEAD_DIM;
    const float *kp = p.k + a0 * (HEADS * HEAD_DIM) + warp * HEAD_DIM, *vp = p.v + a0 * (HEADS * HEAD_DIM) + warp * HEAD_DIM;
    const HeadOperands qk = head_operands(p.q + my_row, kp, n, 0, lane), gv = head_operands(p.gout + my_row, vp, n, 0, lane);
    // ---- the row's first vectors on their way
    const RowHeads hd = row_heads(p.a[(a0 + i) * HEADS + g], p.rule, p.rvlen != nullptr ? p.rvlen + 3ll * tile.x : nullptr,
                                  make_int4(place.z, place.w, 0, 0), p.par);
    const bool mine_here = warp < rows && p.left[a0 + i] == 0;
    const int pairs = n * (n + 1) / 2, slot_bytes = 64 * p.par.tiles;
    int variant = __shfl_sync(FULL, hd.variant, 0);
    auto vectors = [&](int v) { return p.slots + (size_t)(unsigned)(v == 0 ? place.x : place.y + (v - 1) * pairs) * slot_bytes; };
    int tiles = min(row_tiles_of(hd, PA_USUAL_LAG, p.par), p.par.tiles);
    KeyRing<STAGES> ring;
    ring.init((unsigned)__cvta_generic_to_shared(smem + warp * RING), i, n, slot_bytes, lane);
    const bool one_box = __all_sync(FULL, hd.variant == variant);
    if (mine_here) ring.start(vectors(variant), 0, one_box ? tiles : min(tiles, PASS), PASS);

    // ---- logits in bits, gout.v, u
    head_products<true>(qk, kp, n, warp, 0, 1, key_tiles, LOG2E, -INFINITY, logits, row_words, lane);
    head_products<true>(gv, vp, n, warp, 0, 1, key_tiles, 1.0f, 0.0f, dvs, row_words, lane);
    if (BASIS) {
        const float bv[4] = {gv.row.x, gv.row.y, gv.row.z, gv.row.w};
        unsigned bh[4], bl[4], b3[4];
        split3_tf32(bv, bh, bl, b3);
        const float *w = p.W + (size_t)(warp * HEAD_DIM + 4 * t) * 64 + g;
#pragma unroll
        for (int bt = 0; bt < 4; ++bt) {
            float ax[4][2];  // channels 4t ... 4t + 3, bins g and g + 8
#pragma unroll
            for (int c = 0; c < 4; ++c) { ax[c][0] = __ldg(w + c * 64 + bt * 16); ax[c][1] = __ldg(w + c * 64 + bt * 16 + 8); }
            float c[4];
            mma_exact(c, {ax[0][0], ax[0][1], ax[1][0], ax[1][1]}, {ax[2][0], ax[2][1], ax[3][0], ax[3][1]}, bh, bl, b3);
            float *o = us + 2 * t * sums_ld + warp * 64 + bt * 16 + g;
            o[0] = c[0]; o[sums_ld] = c[1]; o[8] = c[2]; o[sums_ld + 8] = c[3];
        }
    }
    if (lane == 0) there[warp] = mine_here ? 1 : 0;
    __syncthreads();

    // ---- a row per warp
    if (mine_here) {
        float4 *lg = reinterpret_cast<float4 *>(logits + warp * row_words) + pa_sum_slot(g, t);
        float4 *dv = reinterpret_cast<float4 *>(dvs + warp * row_words) + pa_sum_slot(g, t);
        float4 *pr = reinterpret_cast<float4 *>(probs + warp * sums_ld) + pa_sum_slot(g, t);
        float4 *gl = reinterpret_cast<float4 *>(glogits + warp * sums_ld) + pa_sum_slot(g, t);
        // the nodes in reach, as the forward chose them
        float top0 = -INFINITY, top1 = -INFINITY;
        for (int T = 0; T < key_tiles; ++T) {
            const float4 l = lg[T * 32];
            top0 = fmaxf(top0, fmaxf(l.x, l.z));
            top1 = fmaxf(top1, fmaxf(l.y, l.w));
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            top0 = fmaxf(top0, __shfl_xor_sync(FULL, top0, o));
            top1 = fmaxf(top1, __shfl_xor_sync(FULL, top1, o));
        }
        const float *own = logits + warp * row_words + (i >> 4) * 128 + ((i >> 3) & 1) * 2;
        const float lag = fmaxf(top0 - own[pa_sum_slot(i & 7, t) * 4], top1 - own[pa_sum_slot(i & 7, t) * 4 + 1]);
        const float most_lag = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(fmaxf(lag, 0.0f))));
        if (most_lag > PA_USUAL_LAG) {
            copy_wait<0>();
            __syncwarp();
            tiles = min(row_tiles_of(hd, most_lag, p.par), p.par.tiles);
            ring.start(vectors(variant), 0, one_box ? tiles : min(tiles, PASS), PASS);
        }
        // delta of head g, from the lane's four channels of it
        const float4 go = __ldg(reinterpret_cast<const float4 *>(p.gout + (a0 + i) * (HEADS * HEAD_DIM)) + lane);
        const float4 ou = __ldg(reinterpret_cast<const float4 *>(p.out + (a0 + i) * (HEADS * HEAD_DIM)) + lane);
        float delta = fmaf(go.w, ou.w, fmaf(go.z, ou.z, fmaf(go.y, ou.y, go.x * ou.x)));
        delta += __shfl_xor_sync(FULL, delta, 1);
        delta += __shfl_xor_sync(FULL, delta, 2);
        const float d0 = __shfl_sync(FULL, delta, 8 * t), d1 = __shfl_sync(FULL, delta, 8 * t + 4);
        const float2 ls = __ldg(reinterpret_cast<const float2 *>(p.lse + (a0 + i) * HEADS + 2 * t));
        const float lse0 = ls.x * LOG2E, lse1 = ls.y * LOG2E;
        // weights (2^-20: the scales of x and rho) and dv - delta in the tables' place
        for (int T = 0; T < key_tiles; ++T) {
            const float4 l = lg[T * 32], d = dv[T * 32];
            lg[T * 32] = make_float4(ex2(l.x - lse0) * 0x1p-20f, ex2(l.y - lse1) * 0x1p-20f, ex2(l.z - lse0) * 0x1p-20f, ex2(l.w - lse1) * 0x1p-20f);
            dv[T * 32] = make_float4(d.x - d0, d.y - d1, d.z - d0, d.w - d1);
        }
        // u of head g as the operand of c (bins x heads), scaled to a largest value between 2^10 and 2^11
        unsigned uh[4][2], ul[4][2];
        float c_scale0 = 1.f, c_scale1 = 1.f;  // c of heads 2t, 2t + 1 from the products
        if (BASIS) {
            float2 u[4][2];
            float most = 0.f;
#pragma unroll
            for (int bt = 0; bt < 4; ++bt)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    u[bt][x] = *reinterpret_cast<const float2 *>(us + warp * sums_ld + g * 64 + bt * 16 + 8 * x + 2 * t);
                    most = fmaxf(most, fmaxf(fabsf(u[bt][x].x), fabsf(u[bt][x].y)));
                }
            most = fmaxf(most, __shfl_xor_sync(FULL, most, 1));
            most = fmaxf(most, __shfl_xor_sync(FULL, most, 2));
            const unsigned e = min(max(__float_as_uint(most) & 0x7f800000u, 30u << 23), 230u << 23);
            const float scale = __uint_as_float((264u << 23) - e), inv = __uint_as_float(e - (10u << 23)) * (1.0f / PG_BASIS_SCALE);
#pragma unroll
            for (int bt = 0; bt < 4; ++bt)
#pragma unroll
                for (int x = 0; x < 2; ++x) split_f16(u[bt][x].x * scale, u[bt][x].y * scale, uh[bt][x], ul[bt][x]);
            c_scale0 = __shfl_sync(FULL, inv, 8 * t);
            c_scale1 = __shfl_sync(FULL, inv, 8 * t + 4);
        }
        if (!one_box) {
            __syncwarp();  // (u has been read)
            for (int T = 0; T < key_tiles; ++T) pr[T * 32] = gl[T * 32] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // The columns are x, x c, x n^2 and x c n^2 (n: nodes from zero), scaled (column_scales)
        const float2 aa = make_float2(__shfl_sync(FULL, hd.a2h2, 8 * t), __shfl_sync(FULL, hd.a2h2, 8 * t + 4));
        const int var0 = __shfl_sync(FULL, hd.variant, 8 * t), var1 = __shfl_sync(FULL, hd.variant, 8 * t + 4);
        float ga0 = 0.f, ga1 = 0.f, m0 = 0.f, m1 = 0.f;  // m: sum_j w S2
        for (int first = 0; first < tiles; first += PASS) {
            const int count = min(PASS, tiles - first);
            unsigned xh[PASS][2], xl[PASS][2], zh[PASS][2], zl[PASS][2], yh[PASS][2], yl[PASS][2], th[PASS][2], tl[PASS][2];
#pragma unroll
            for (int u = 0; u < PASS; ++u) {
                if (u >= count) break;
                const int mt = first + u;
                const float n0 = (float)(mt * PG_TILE - PG_BELOW + g), n1 = n0 + 8.0f, q0 = n0 * n0, q1 = n1 * n1;
                const float2 e0 = mul2(aa, make_float2(q0, q0)), e1 = mul2(aa, make_float2(q1, q1));
                float x[4] = {ex2(e0.x) * PA_W_SCALE, ex2(e0.y) * PA_W_SCALE, ex2(e1.x) * PA_W_SCALE, ex2(e1.y) * PA_W_SCALE};
                const float s0 = q0 * p.n2_scale, s1 = q1 * p.n2_scale;
                node_operand(x, xh[u], xl[u]);
                const float z[4] = {x[0] * s0, x[1] * s0, x[2] * s1, x[3] * s1};
                node_operand(z, zh[u], zl[u]);
                if (BASIS) {
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int bt = 0; bt < 4; ++bt) {
                        const int2 reach = node_tiles_in_reach(bt, p.inv_wscale);
                        if (mt < reach.x || mt >= reach.y) continue;
                        const uint4 gh = __ldg(p.basis_nodes + (size_t)(mt * 4 + bt) * 64 + lane), gl4 = __ldg(p.basis_nodes + (size_t)(mt * 4 + bt) * 64 + 32 + lane);
                        float b[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_f16(b, gl4.x, gl4.y, gl4.z, gl4.w, uh[bt][0], uh[bt][1]);
                        mma_f16(b, gh.x, gh.y, gh.z, gh.w, ul[bt][0], ul[bt][1]);
                        mma_f16(b, gh.x, gh.y, gh.z, gh.w, uh[bt][0], uh[bt][1]);
#pragma unroll
                        for (int w = 0; w < 4; ++w) c[w] += b[w];
                    }
#pragma unroll
                    for (int w = 0; w < 4; ++w) c[w] *= x[w] * p.c_scale;
                    node_operand(c, yh[u], yl[u]);
                    const float tt[4] = {c[0] * s0, c[1] * s0, c[2] * s1, c[3] * s1};
                    node_operand(tt, th[u], tl[u]);
                }
            }
            bool open = true;  // this lane's head g waits for its variant
            while (true) {
                const bool mine0 = var0 == variant, mine1 = var1 == variant;
                for (int T = 0; T < key_tiles; ++T) {
                    float S0[4] = {0.f, 0.f, 0.f, 0.f}, low[4] = {0.f, 0.f, 0.f, 0.f}, S1[4] = {0.f, 0.f, 0.f, 0.f}, S2[4] = {0.f, 0.f, 0.f, 0.f}, S3[4] = {0.f, 0.f, 0.f, 0.f};
                    const unsigned plain = ring.plain + ring.take();
#pragma unroll
                    for (int u = 0; u < PASS; ++u) {
                        if (u >= count) break;
                        unsigned hi[4], lo[4];
                        ldmatrix4(lo, plain + u * 64 + 32);
                        ldmatrix4(hi, plain + u * 64);
                        mma_f16(low, lo[0], lo[1], lo[2], lo[3], xh[u][0], xh[u][1]);
                        mma_f16(S2, lo[0], lo[1], lo[2], lo[3], zh[u][0], zh[u][1]);
                        if (BASIS) {
                            mma_f16(S1, lo[0], lo[1], lo[2], lo[3], yh[u][0], yh[u][1]);
                            mma_f16(S3, lo[0], lo[1], lo[2], lo[3], th[u][0], th[u][1]);
                        }
                        mma_f16(low, hi[0], hi[1], hi[2], hi[3], xl[u][0], xl[u][1]);
                        mma_f16(S2, hi[0], hi[1], hi[2], hi[3], zl[u][0], zl[u][1]);
                        if (BASIS) {
                            mma_f16(S1, hi[0], hi[1], hi[2], hi[3], yl[u][0], yl[u][1]);
                            mma_f16(S3, hi[0], hi[1], hi[2], hi[3], tl[u][0], tl[u][1]);
                        }
                        mma_f16(S0, hi[0], hi[1], hi[2], hi[3], xh[u][0], xh[u][1]);
                        mma_f16(S2, hi[0], hi[1], hi[2], hi[3], zh[u][0], zh[u][1]);
                        if (BASIS) {
                            mma_f16(S1, hi[0], hi[1], hi[2], hi[3], yh[u][0], yh[u][1]);
                            mma_f16(S3, hi[0], hi[1], hi[2], hi[3], th[u][0], th[u][1]);
                        }
                    }
                    ring.done();
#pragma unroll
                    for (int c = 0; c < 4; ++c) S0[c] += low[c];
                    float4 w = lg[T * 32];
                    const float4 d = dv[T * 32];
                    if (!one_box) { w.x = mine0 ? w.x : 0.f; w.z = mine0 ? w.z : 0.f; w.y = mine1 ? w.y : 0.f; w.w = mine1 ? w.w : 0.f; }
                    const float4 pp = make_float4(w.x * S0[0], w.y * S0[1], w.z * S0[2], w.w * S0[3]);
                    float4 gg = make_float4(pp.x * d.x, pp.y * d.y, pp.z * d.z, pp.w * d.w);
                    const float4 ww = make_float4(w.x * S2[0], w.y * S2[1], w.z * S2[2], w.w * S2[3]);
                    m0 += ww.x + ww.z;
                    m1 += ww.y + ww.w;
                    ga0 += fmaf(ww.x, d.x, ww.z * d.z);
                    ga1 += fmaf(ww.y, d.y, ww.w * d.w);
                    if (BASIS) {
                        const float k0 = c_scale0 * p.c_unit, k1 = c_scale1 * p.c_unit;
                        gg.x = fmaf(w.x * k0, S1[0], gg.x); gg.y = fmaf(w.y * k1, S1[1], gg.y);
                        gg.z = fmaf(w.z * k0, S1[2], gg.z); gg.w = fmaf(w.w * k1, S1[3], gg.w);
                        ga0 = fmaf(w.x * k0, S3[0], fmaf(w.z * k0, S3[2], ga0));
                        ga1 = fmaf(w.y * k1, S3[1], fmaf(w.w * k1, S3[3], ga1));
                    }
                    if (first == 0 && one_box) {
                        pr[T * 32] = pp;
                        gl[T * 32] = gg;
                    } else {
                        const float4 a = pr[T * 32], b = gl[T * 32];
                        pr[T * 32] = make_float4(a.x + pp.x, a.y + pp.y, a.z + pp.z, a.w + pp.w);
                        gl[T * 32] = make_float4(b.x + gg.x, b.y + gg.y, b.z + gg.z, b.w + gg.w);
                    }
                }
                if (one_box) break;  // (the ring runs on to the next pass)
                open = open && hd.variant != variant;
                const unsigned left = __ballot_sync(FULL, open);
                copy_wait<0>();
                __syncwarp();
                variant = __shfl_sync(FULL, hd.variant, left != 0u ? __ffs(left) - 1 : 0);
                const int from = left != 0u ? first : first + PASS;
                if (from < tiles) ring.start(vectors(variant), from, min(tiles - from, PASS), PASS);
                if (left == 0u) break;
            }
        }
        copy_wait<0>();
        // The probabilities' own sum takes what lse and the sums of the forward are off by out of them and of all that is
        // proportional to them (one key: exactly 1, and v's gradient that of its output), the gradients' own sum what delta is off
        float sum0 = 0.f, sum1 = 0.f, off0 = 0.f, off1 = 0.f;
        for (int T = 0; T < key_tiles; ++T) {
            const float4 a = pr[T * 32], b = gl[T * 32];
            sum0 += a.x + a.z;
            sum1 += a.y + a.w;
            off0 += b.x + b.z;
            off1 += b.y + b.w;
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            ga0 += __shfl_xor_sync(FULL, ga0, o);
            ga1 += __shfl_xor_sync(FULL, ga1, o);
            m0 += __shfl_xor_sync(FULL, m0, o);
            m1 += __shfl_xor_sync(FULL, m1, o);
            sum0 += __shfl_xor_sync(FULL, sum0, o);
            sum1 += __shfl_xor_sync(FULL, sum1, o);
            off0 += __shfl_xor_sync(FULL, off0, o);
            off1 += __shfl_xor_sync(FULL, off1, o);
        }
        off0 = -off0 / sum0;
        off1 = -off1 / sum1;
        if (g == 0) *reinterpret_cast<float2 *>(p.ga + (a0 + i) * HEADS + 2 * t) = make_float2(fmaf(off0, m0, ga0) / sum0 * p.ga_unit, fmaf(off1, m1, ga1) / sum1 * p.ga_unit);
        // per edge, for the sums over the rows
        float2 *po = reinterpret_cast<float2 *>(p.prob + (e0 + g) * HEADS + 2 * t), *go2 = reinterpret_cast<float2 *>(p.glogit + (e0 + g) * HEADS + 2 * t);
        const float norm0 = 1.0f / sum0, norm1 = 1.0f / sum1;
        for (int T = 0; T < key_tiles; ++T) {
            const int j = T * PA_KEYS + g;
            const float4 a = pr[T * 32];
            float4 b = gl[T * 32];
            b = make_float4(fmaf(off0, a.x, b.x) * norm0, fmaf(off1, a.y, b.y) * norm1, fmaf(off0, a.z, b.z) * norm0, fmaf(off1, a.w, b.w) * norm1);
            gl[T * 32] = b;
            const size_t at = (size_t)T * PA_KEYS * HEADS / 2;
            if (j < n) { po[at] = make_float2(a.x / sum0, a.y / sum1); go2[at] = make_float2(b.x, b.y); }
            if (j + 8 < n) { po[at + 4 * HEADS] = make_float2(a.z / sum0, a.w / sum1); go2[at + 4 * HEADS] = make_float2(b.z, b.w); }
        }
    }
    __syncthreads();

    // ---- gq: C[channel][row] of head `warp`, sixteen keys at a time in the order 2t, 2t + 1, 2t + 8, 2t + 9
    {
        const float *k0 = kp + g;
        const bool in = there[g] != 0;
        const float *gr = glogits + g * sums_ld + (warp & 1);
        const int slot0 = pa_sum_slot(2 * t, warp >> 1) * 4, slot1 = pa_sum_slot(2 * t + 1, warp >> 1) * 4;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int T = 0; T < key_tiles; ++T) {
            float kk[4][2];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float *at = k0 + min(T * PA_KEYS + 2 * t + (u & 1) + 8 * (u >> 1), n - 1) * (HEADS * HEAD_DIM);
                kk[u][0] = __ldg(at);
                kk[u][1] = __ldg(at + 8);
            }
            const float *gt = gr + T * 128;
            const float bv[4] = {in ? gt[slot0] : 0.f, in ? gt[slot1] : 0.f, in ? gt[slot0 + 2] : 0.f, in ? gt[slot1 + 2] : 0.f};
            unsigned bh[4], bl[4], b3[4];
            split3_tf32(bv, bh, bl, b3);
            float c[4];
            mma_exact(c, {kk[0][0], kk[0][1], kk[1][0], kk[1][1]}, {kk[2][0], kk[2][1], kk[3][0], kk[3][1]}, bh, bl, b3);
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] += c[u];
        }
        float *o = p.gq + (a0 + i0 + 2 * t) * (HEADS * HEAD_DIM) + warp * HEAD_DIM + g;
        if (there[2 * t]) { o[0] = acc[0]; o[8] = acc[2]; }
        if (there[2 * t + 1]) { o[128] = acc[1]; o[136] = acc[3]; }
    }
}

}  // namespace

int launch_pair_attn_bwd(const PairAttn &l, cudaStream_t s)
{
    if (l.N == 0) return CF_OK;
    Args p{};
    p.q = l.q; p.k = l.k; p.v = l.v; p.a = l.a; p.rvlen = l.rvlen; p.W = l.W; p.out = l.out; p.gout = l.gout; p.lse = l.lse;
    p.edge_start = l.edge_start; p.rule = l.rule; p.par = l.par; p.slots = l.grid.slots; p.tiles = l.grid.tiles; p.counters = l.grid.counters;
    p.left = l.left; p.basis_nodes = l.grid.basis_nodes;
    p.inv_wscale = l.wscale > 0 ? (float)(1.0 / (double)(float)l.wscale) : 1.0f;
    column_scales(p, (double)(float)l.wscale);
    p.gq = l.gq; p.ga = l.ga; p.glogit = l.glogit; p.prob = l.prob; p.max_atoms = l.max_atoms;
    auto kernel = l.K > 0 ? pair_attn_bwd_kernel<true> : pair_attn_bwd_kernel<false>;
    static thread_local bool configured[64][2] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    bool &done = configured[dev & 63][l.K > 0 ? 1 : 0];
    if (!done) {
        const size_t most = smem_bytes(PG_MAX_ATOMS, l.K > 0);
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) {
            cudaGetLastError();
            return fail(CF_ERR_CUDA, "pair attention, backward: %zu bytes of shared memory not available", most);
        }
        done = true;
    }
    kernel<<<(unsigned)(l.N / PG_ROWS + l.B), THREADS, smem_bytes(l.max_atoms, l.K > 0), s>>>(p);
    return launch_status("pair_attn_bwd_kernel");
}

}  // namespace cf
