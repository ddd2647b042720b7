// Infinitely connected attention over pair grids (pair_grid.cuh), forward.
//
// With rho_j the vector of the pair (i, j), x_h[m] = exp(a_h d_m^2) and w_h[j] = exp(q_i.k_j - max), a row of the attention is
//     S_h[j] = sum_m rho_j[m] x_h[m]        p_h[j] = w_h[j] S_h[j] / Z_h        Z_h = sum_j w_h[j] S_h[j] = sum_m E_h[m]
//     E_h[m] = x_h[m] sum_j w_h[j] rho_j[m]       Psi_h[k] = sum_m E_h[m] g_k(d_m) / Z_h
//     out_h  = sum_j p_h[j] v_j + W_h Psi_h
// whatever the number of images: two products of the (keys x nodes) matrix rho with eight columns, one of them transposed.
//
// Block = eight rows of a crystal.  (1) warp = head: the logits of the eight rows, one product.  (2) warp = row: the products
// with rho, 16 keys x 48 nodes at a time through shared memory, which serves both orientations (ldmatrix plain and transposed),
// in passes of up to six node tiles whose sums a warp holds in registers.  (3) warp = head again: sum p v, and E of the eight rows
// times the projected basis (TAIL = PROJECTED: W_h g(d_m), made once per call), or Psi, which the backward needs, and its
// projection (TAIL = KEEP_PSI).  Operands are half pairs (nodes, weights: scaled by 2^15, exact to 22 bits over the range that
// matters), three products each with the small ones first, or three TF32 pieces where the range is the caller's (q, k, v, W, w S).
// (Logits and sum p v by a row's own warp, with float32 sums, cost 10-20 % more: keys and values then come through the L1 once per
// row instead of once per block.)
//
// Bound: latency at sixteen warps on an SM (128 registers, 95-113 KB of tables and rings).  1,024 crystals of up to 60 atoms 309 us
// per call under ncu, issue slots 42 %, LSU wavefronts 47 %, tensor pipe 24 %, DRAM 1.7 TB/s; 128 of up to 30 34 us, 31, 19, 14 %.
// The scales per head and the rows' own sum for lse (see there) took the former from 306.
#include <initializer_list>

#include "pair_attn.cuh"

namespace cf {
int launch_leftover_rows(const float *q, const float *k, const float *v, const float *a, const float *pos_ij,
                         const float *tvecs, const float *rvlen, const int64_t *batch, const int64_t *edges,
                         const int64_t *row_start, int64_t N, int64_t E, int64_t max_atoms, double dist_max,
                         double wscale, const float *W, double cutoff_radius, int lattice_range, int minimum_range,
                         float *out, float *logit, float *lse, float *psi_row, const int *rows, const unsigned *count,
                         unsigned *ticket, int64_t K, cudaStream_t s);
namespace {

constexpr int PASS = 6;  // node tiles of a pass
static_assert(PG_TILES_BASIS <= 2 * PASS && PG_TILES_PLAIN <= PASS && PASS == 2 * PA_STEP, "two passes of two steps");
constexpr int PSI_LD = 512 + 20;
constexpr int E_ROW = PASS * 512 + 64;  // bytes of a row's E of the first pass

enum Tail { PLAIN, PROJECTED, KEEP_PSI };  // no basis; inference; training

// Shared memory of a block: a ring per warp (which the last E, then Psi take over), E of the first pass,
// the rows' logits / weights and their sums S.
template <int TAIL, int STAGES>
struct Layout {
    static constexpr int WARPS = PG_ROWS, THREADS = 32 * WARPS;
    // (rows 64 mod 128 bytes apart, for the reads of eight rows at a time)
    static constexpr int REGION = (KeyRing<STAGES>::BYTES + 127) / 128 * 128 + 64;
    static constexpr int E_BYTES = TAIL != PLAIN ? PG_ROWS * E_ROW : 0;
    static constexpr int TABLES = WARPS * REGION + E_BYTES;
    static_assert(PASS * 512 <= REGION, "E of a pass fits a ring");
    static_assert(PG_ROWS * PSI_LD * 4 <= WARPS * REGION, "Psi fits the rings");
    static size_t bytes(int max_atoms) { return TABLES + 2 * sizeof(float) * PG_ROWS * pa_row_words(max_atoms); }
};

struct Args {
    const float *q, *k, *v, *a, *rvlen, *W;
    const int64_t *atom_start, *edge_start;
    BoxRule rule;
    PairGridParams par;
    const unsigned char *slots;
    const int4 *tiles;
    unsigned *counters;   // counters[0]: tiles
    unsigned *left_count;
    int *leftover;
    unsigned char *left;
    const uint4 *basis, *projected;
    const float *projected_scale;
    float inv_wscale;
    float *out, *lse, *psi_row;
    int max_atoms;
    unsigned long long *stats;  // { -, -, rows, products of 16 keys x 16 nodes } added up, or null
};

struct Row {
    float *weights, *sums;        // tables
    int key_tiles, n, pairs, slot_first, extra_first, slot_bytes;
    const unsigned char *slots;
    int variant;                  // the ring's
    __device__ __forceinline__ const unsigned char *vectors() const
    {
        return slots + (size_t)(unsigned)(variant == 0 ? slot_first : extra_first + (variant - 1) * pairs) * slot_bytes;
    }
};

// One pass: N node tiles from `first`.  S of all keys into the table (`fresh`: what it held does not count), E = x sum_j w rho in
// E.
// PER_TILE: a node tile's large products have a sum of their own, added in registers.
template <bool PER_TILE, int N, int STAGES>
__device__ __forceinline__ void node_pass(Row &row, KeyRing<STAGES> &ring, bool fresh, int first, const RowHeads &hd, int lane, float (&E)[PASS][4],
                                          float2 &z, float2 &largest)
{
    const int g = lane >> 2, t = lane & 3;
    const float a2h2 = hd.a2h2;
    unsigned xh[N][2], xl[N][2];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        E[u][0] = E[u][1] = E[u][2] = E[u][3] = 0.f;
        const float m = (float)((first + u) * PG_TILE - PG_BELOW + 2 * t);
        const float2 x0 = mul2(gauss2(a2h2, m), make_float2(PA_W_SCALE, PA_W_SCALE));
        const float2 x1 = mul2(gauss2(a2h2, m + 8.0f), make_float2(PA_W_SCALE, PA_W_SCALE));
        split_f16(x0.x, x0.y, xh[u][0], xl[u][0]);
        split_f16(x1.x, x1.y, xh[u][1], xl[u][1]);
    }
    const int var0 = __shfl_sync(FULL, hd.variant, 8 * t), var1 = __shfl_sync(FULL, hd.variant, 8 * t + 4);
    bool open = true;  // this lane's head g waits for its variant
    while (true) {
        const bool mine = hd.variant == row.variant, mine0 = var0 == row.variant, mine1 = var1 == row.variant;
        float4 *o = reinterpret_cast<float4 *>(row.sums) + pa_sum_slot(g, t);
        const uint4 *wp = reinterpret_cast<const uint4 *>(row.weights) + lane;
        for (int T = 0; T < row.key_tiles; ++T, o += 32, wp += 32) {
            uint4 w = *wp;
            if (!mine) w = make_uint4(0u, 0u, 0u, 0u);
            // (the tensor pipe truncates what it adds to: the small products have a sum of their own, and what it cut off the large ones'
            // last addition is given back)
            float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f}, small[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int f = 0; f < N; f += PA_STEP) {
                const unsigned at = ring.take(), plain = ring.plain + at, trans = ring.trans + at;
#pragma unroll
                for (int u = f; u < f + PA_STEP && u < N; ++u) {
                    float(&sum)[4] = u & 1 ? sb : sa;
                    unsigned hi[4], lo[4];
                    ldmatrix4(lo, plain + (u - f) * 64 + 32);
                    ldmatrix4(hi, plain + (u - f) * 64);
                    mma_f16(small, lo[0], lo[1], lo[2], lo[3], xh[u][0], xh[u][1]);
                    mma_f16(small, hi[0], hi[1], hi[2], hi[3], xl[u][0], xl[u][1]);
                    if (PER_TILE) {
                        float c[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_f16(c, hi[0], hi[1], hi[2], hi[3], xh[u][0], xh[u][1]);
#pragma unroll
                        for (int x = 0; x < 4; ++x) sum[x] += c[x];
                    } else {
                        mma_f16(sum, hi[0], hi[1], hi[2], hi[3], xh[u][0], xh[u][1]);
                    }
                    ldmatrix4_trans(lo, trans + (u - f) * 64 + 32);
                    ldmatrix4_trans(hi, trans + (u - f) * 64);
                    mma_f16(E[u], lo[0], lo[1], lo[2], lo[3], w.x, w.y);
                    mma_f16(E[u], hi[0], hi[1], hi[2], hi[3], w.z, w.w);
                    mma_f16(E[u], hi[0], hi[1], hi[2], hi[3], w.x, w.y);
                }
                ring.done();
            }
            // S of keys g and g + 8, heads 2t and 2t + 1
            auto whole = [&](int x) {
                const float large = sb[x] + sa[x];
                return large + fmaf(large, MMA_LOST, small[x]);
            };
            float4 sum = make_float4(whole(0), whole(1), whole(2), whole(3));
            if (!fresh) {
                const float4 v = *o;
                sum = make_float4(v.x + (mine0 ? sum.x : 0.f), v.y + (mine1 ? sum.y : 0.f), v.z + (mine0 ? sum.z : 0.f), v.w + (mine1 ? sum.w : 0.f));
            }
            *o = sum;
        }
        open = open && !mine;
        const unsigned left = __ballot_sync(FULL, open);
        if (left == 0u) break;
        copy_wait<0>();
        __syncwarp();
        row.variant = __shfl_sync(FULL, hd.variant, __ffs(left) - 1);
        ring.start(row.vectors(), first, N, PASS);
    }
    // heads 2t and 2t + 1 at nodes g and g + 8 of a tile
    const float2 aa = make_float2(__shfl_sync(FULL, a2h2, 8 * t), __shfl_sync(FULL, a2h2, 8 * t + 4));
    float2 most = make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const float n0 = (float)((first + u) * PG_TILE - PG_BELOW + g), n1 = n0 + 8.0f;
        const float2 e0 = mul2(aa, make_float2(n0 * n0, n0 * n0)), e1 = mul2(aa, make_float2(n1 * n1, n1 * n1));
        const float2 r0 = mul2(make_float2(E[u][0], E[u][1]), make_float2(ex2(e0.x), ex2(e0.y)));
        const float2 r1 = mul2(make_float2(E[u][2], E[u][3]), make_float2(ex2(e1.x), ex2(e1.y)));
        E[u][0] = r0.x; E[u][1] = r0.y; E[u][2] = r1.x; E[u][3] = r1.y;
        z = add2(z, add2(r0, r1));
        most = make_float2(fmaxf(most.x, fmaxf(fabsf(r0.x), fabsf(r1.x))), fmaxf(most.y, fmaxf(fabsf(r0.y), fabsf(r1.y))));
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) most = make_float2(fmaxf(most.x, __shfl_xor_sync(FULL, most.x, o)), fmaxf(most.y, __shfl_xor_sync(FULL, most.y, o)));
    largest = most;
}

// E as the operand of the product with the basis (nodes x heads), half pairs; scales of heads 2t, 2t + 1
template <int N>
__device__ __forceinline__ void store_e(const float (&E)[PASS][4], float2 scale, unsigned char *at, int lane)
{
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const float2 r0 = mul2(make_float2(E[u][0], E[u][1]), scale), r1 = mul2(make_float2(E[u][2], E[u][3]), scale);
        unsigned h0, l0, h1, l1;
        split_f16(r0.x, r0.y, h0, l0);
        split_f16(r1.x, r1.y, h1, l1);
        reinterpret_cast<uint4 *>(at)[u * 32 + lane] = make_uint4(transpose_8x8(h0), transpose_8x8(h1), transpose_8x8(l0), transpose_8x8(l1));
    }
}

// f<N>() for N = count, 1 ... PASS
#define BY_TILES(count, ...)                                                            \
    switch (count) {                                                                    \
    case 1: { constexpr int N = 1; __VA_ARGS__ } break;                                 \
    case 2: { constexpr int N = 2; __VA_ARGS__ } break;                                 \
    case 3: { constexpr int N = 3; __VA_ARGS__ } break;                                 \
    case 4: { constexpr int N = 4; __VA_ARGS__ } break;                                 \
    case 5: { constexpr int N = 5; __VA_ARGS__ } break;                                 \
    case 6: { constexpr int N = 6; __VA_ARGS__ } break;                                 \
    default: break;                                                                     \
    }

template <int TAIL, int STAGES>
__global__ void __launch_bounds__(Layout<TAIL, STAGES>::THREADS, 2) pair_attn_kernel(const Args p)
{
    extern __shared__ __align__(128) unsigned char smem[];
    using L = Layout<TAIL, STAGES>;
    constexpr bool BASIS = TAIL != PLAIN;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(FULL, tid >> 5, 0), g = lane >> 2, t = lane & 3;
    const int row_words = pa_row_words(p.max_atoms);
    float *tables = reinterpret_cast<float *>(smem + L::TABLES), *sums = tables + PG_ROWS * row_words;
    __shared__ float e_unit[PG_ROWS][HEADS], tops[PG_ROWS][HEADS];  // one of E as stored, over Z; largest logits
    __shared__ int row_tiles[PG_ROWS];  // node tiles of a row; 0: it is not there or left over
    __shared__ unsigned odd[PG_ROWS];   // 1: a row's result is not finite
    grid_launch_dependents();
    grid_dependency_wait();  // q, k, v, a
    const int4 tile = p.tiles[2 * blockIdx.x], place = p.tiles[2 * blockIdx.x + 1];
    if (blockIdx.x >= p.counters[0]) return;
    const int i0 = tile.y, n = abs(tile.z), rows = min(PG_ROWS, n - i0);
    const long long a0 = tile.w;
    if (tile.z < 0 || n > p.max_atoms) {  // no vectors, or more atoms than the caller said: the row kernel's
        if (tid < rows) {
            p.leftover[atomicAdd(p.left_count, 1u)] = (int)(a0 + i0 + tid);
            if (p.left != nullptr) p.left[a0 + i0 + tid] = 1;
        }
        return;
    }
    Row row;
    row.key_tiles = (n + PA_KEYS - 1) / PA_KEYS; row.n = n; row.pairs = n * (n + 1) / 2; row.slot_first = place.x; row.extra_first = place.y;
    row.slot_bytes = 64 * p.par.tiles; row.slots = p.slots;
    row.weights = tables + warp * row_words; row.sums = sums + warp * row_words;

    const HeadOperands ops = head_operands(p.q + (a0 + min(i0 + g, n - 1)) * (HEADS * HEAD_DIM) + warp * HEAD_DIM,
                                           p.k + a0 * (HEADS * HEAD_DIM) + warp * HEAD_DIM, n, 0, lane);
    // ---- the row's first vectors on their way
    const int i = i0 + min(warp, rows - 1);
    const RowHeads hd = row_heads(p.a[(a0 + i) * HEADS + g], p.rule, p.rvlen != nullptr ? p.rvlen + 3ll * tile.x : nullptr,
                                  make_int4(place.z, place.w, 0, 0), p.par);
    int tiles = row_tiles_of(hd, PA_USUAL_LAG, p.par), count = 0;  // of the row; of its first pass
    bool good = !__any_sync(FULL, hd.variant < 0 || hd.narrow) && tiles <= p.par.tiles && warp < rows;
    row.variant = __shfl_sync(FULL, hd.variant, 0);
    const bool one_box = __all_sync(FULL, hd.variant == row.variant);
    KeyRing<STAGES> ring;
    ring.init((unsigned)__cvta_generic_to_shared(smem + warp * L::REGION), i, n, row.slot_bytes, lane);
    auto start = [&]() {
        count = min(tiles, PASS);
        ring.start(row.vectors(), 0, one_box ? tiles : count, PASS);
    };
    if (good) start();

    // ---- logits in bits
    head_products<false>(ops, p.k + a0 * (HEADS * HEAD_DIM) + warp * HEAD_DIM, n, warp, 0, 1, row.key_tiles, LOG2E, -INFINITY, tables, row_words, lane);
    __syncthreads();

    // ---- a row per warp, or half of one
    float top = 0.f;
    if (good) {
        top = row_top(row.weights, row.key_tiles, lane);
        // (the logit of the row's own atom, from the lane that has it)
        const float own = row.weights[(i >> 4) * 128 + pa_key_word(g, i & 7) + ((i >> 3) & 1) * 2];
        const float lag = top - own;
        good = __all_sync(FULL, lag <= PA_MAX_LAG);
        if (good && __any_sync(FULL, lag > PA_USUAL_LAG)) {  // nodes further out: from the beginning
            copy_wait<0>();
            __syncwarp();
            tiles = row_tiles_of(hd, lag, p.par);
            good = tiles <= p.par.tiles;
            if (good) start();
        }
    }
    if (good) weights_in_place(row.weights, row.key_tiles, top, lane);
    __syncwarp();
    float2 z = make_float2(0.f, 0.f);
    if (good) {
        float E[PASS][4];
        float2 largest, unit = make_float2(1.f, 1.f);
        if (!one_box) {
            for (int T = 0; T < row.key_tiles; ++T) reinterpret_cast<float4 *>(row.sums)[T * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            __syncwarp();
        }
        BY_TILES(count, node_pass<!BASIS, N>(row, ring, one_box, 0, hd, lane, E, z, largest);)
        if (BASIS) {
            // every head scaled to a largest value between 2^10 and 2^11: the second pass has 2^5 to exceed the first.  (One scale for the
            // row left 20 bits to a head 2^15 below the others: 1e-6 of its sums.)
            auto exponent = [](float v) { return min(max(__float_as_uint(v) & 0x7f800000u, 30u << 23), 230u << 23); };
            const unsigned x0 = exponent(largest.x), x1 = exponent(largest.y);
            const float2 scale = make_float2(__uint_as_float((264u << 23) - x0), __uint_as_float((264u << 23) - x1));
            unit = make_float2(__uint_as_float(x0 - (10u << 23)), __uint_as_float(x1 - (10u << 23)));
            BY_TILES(count, store_e<N>(E, scale, smem + L::WARPS * L::REGION + warp * E_ROW, lane);)
            const int more = tiles - count;
            if (more > 0) {
                if (!one_box) {
                    copy_wait<0>();
                    __syncwarp();
                    row.variant = __shfl_sync(FULL, hd.variant, 0);
                    ring.start(row.vectors(), PASS, more, PASS);
                }
                BY_TILES(more, node_pass<!BASIS, N>(row, ring, false, PASS, hd, lane, E, z, largest); copy_wait<0>(); __syncwarp();
                         store_e<N>(E, scale, smem + warp * L::REGION, lane);)
                good = __all_sync(FULL, largest.x * scale.x < 60000.0f && largest.y * scale.y < 60000.0f);
            }
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            z.x += __shfl_xor_sync(FULL, z.x, o);
            z.y += __shfl_xor_sync(FULL, z.y, o);
        }
        if (BASIS && g == 0) *reinterpret_cast<float2 *>(&e_unit[warp][2 * t]) = make_float2(unit.x / z.x, unit.y / z.y);
    }
    copy_wait<0>();
    // (an infinity or a NaN anywhere in the row, or sums that overflow: the row kernel's)
    good = good && __all_sync(FULL, z.x > 1e-30f && z.x < 1e30f && z.y > 1e-30f && z.y < 1e30f);
    if (t == 0) tops[warp][g] = top;
    if (lane == 0) {
        odd[warp] = 0u;
        row_tiles[warp] = good ? tiles : 0;
        if (p.stats != nullptr && good) {
            atomicAdd(p.stats + 2, 1ull);
            atomicAdd(p.stats + 3, (unsigned long long)(row.key_tiles * tiles));
        }
        if (warp < rows) {
            if (!good) p.leftover[atomicAdd(p.left_count, 1u)] = (int)(a0 + i);
            if (p.left != nullptr) p.left[a0 + i] = good ? 0 : 1;
        }
    }
    const int h = warp;
    const float *vp = p.v + a0 * (HEADS * HEAD_DIM) + h * HEAD_DIM + g;
    float v[4][2];
    auto load_values = [&](int T) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float *at = vp + min(T * PA_KEYS + 2 * t + (u & 1) + 8 * (u >> 1), n - 1) * (HEADS * HEAD_DIM);
            v[u][0] = __ldg(at);
            v[u][1] = __ldg(at + 8);
        }
    };
    load_values(0);
    __syncthreads();

    // ---- values: C[channel][row] of head h; the keys in the order of the tables, loaded a tile ahead
    const int tiles_g = row_tiles[g];
    const bool in0 = row_tiles[2 * t] > 0, in1 = row_tiles[2 * t + 1] > 0;
    float val[4] = {0.f, 0.f, 0.f, 0.f}, total0, total1;
    {
        const uint4 *wp = reinterpret_cast<const uint4 *>(tables + g * row_words) + h * 4 + t;
        const float4 *sp = reinterpret_cast<const float4 *>(sums + g * row_words);
        const int slot0 = pa_sum_slot(2 * t, h >> 1), slot1 = pa_sum_slot(2 * t + 1, h >> 1);
        const bool second = (h & 1) != 0;
        float total = 0.f;
        for (int T = 0; T < row.key_tiles; ++T) {
            const float va[4] = {v[0][0], v[0][1], v[1][0], v[1][1]}, vb[4] = {v[2][0], v[2][1], v[3][0], v[3][1]};
            if (T + 1 < row.key_tiles) load_values(T + 1);
            const float4 w = weights_of(wp[T * 32]), s0 = sp[T * 32 + slot0], s1 = sp[T * 32 + slot1];
            float4 b = make_float4(w.x * (second ? s0.y : s0.x), w.y * (second ? s1.y : s1.x), w.z * (second ? s0.w : s0.z), w.w * (second ? s1.w : s1.z));
            if (tiles_g <= 0) b = make_float4(0.f, 0.f, 0.f, 0.f);
            total += (b.x + b.y) + (b.z + b.w);
            // (a sum of its own per key tile, added in registers)
            const float bv[4] = {b.x, b.y, b.z, b.w};
            unsigned bh[4], bl[4], b3[4];
            split3_tf32(bv, bh, bl, b3);
            float c[4];
            mma_exact(c, va, vb, bh, bl, b3);
#pragma unroll
            for (int u = 0; u < 4; ++u) val[u] += c[u];
        }
        // divided by the sum of these very weights, of row g in the lanes of g
        total += __shfl_xor_sync(FULL, total, 1);
        total += __shfl_xor_sync(FULL, total, 2);
        // (their sum is closer than Z, which the tensor pipe adds key tile by key tile; scales: weights and Gaussians 2^15, vectors 2^5)
        if (p.lse != nullptr && t == 0 && tiles_g > 0) p.lse[(a0 + i0 + g) * HEADS + h] = (tops[g][h] + log2f(total * 0x1p-35f)) * LN2;
        total0 = __shfl_sync(FULL, total, 8 * t);
        total1 = __shfl_sync(FULL, total, 8 * t + 4);
        const float f0 = in0 ? 1.0f / total0 : 0.f, f1 = in1 ? 1.0f / total1 : 0.f;
        val[0] *= f0; val[1] *= f1; val[2] *= f0; val[3] *= f1;
    }
    float proj[4] = {0.f, 0.f, 0.f, 0.f};
    float *ps = reinterpret_cast<float *>(smem);  // Psi
    const unsigned char *eg0 = smem + L::WARPS * L::REGION + g * E_ROW + t * 16;
    const unsigned char *eg1 = smem + g * L::REGION + t * 16 - PASS * 512;
    auto e_of = [&](int mt, int head) {  // E of row g in a head, as the operand (nodes x rows)
        return mt < tiles_g ? *reinterpret_cast<const uint4 *>((mt < PASS ? eg0 : eg1) + mt * 512 + head * 64) : make_uint4(0u, 0u, 0u, 0u);
    };
    const int most_tiles = (int)__reduce_max_sync(FULL, (unsigned)tiles_g);
    if (TAIL == PLAIN) {
    } else if (TAIL == PROJECTED) {
        // ---- sum_m V_h[m] E[m], the fragments a tile ahead
        const uint4 *frag = p.projected + (size_t)h * PG_TILES_BASIS * 64 + lane;
        int mt = 0;
        uint4 vh = make_uint4(0u, 0u, 0u, 0u), vl = vh;
        if (mt < most_tiles) { vh = __ldg(frag + mt * 64); vl = __ldg(frag + mt * 64 + 32); }
        for (; mt < most_tiles; ++mt) {
            const uint4 ch = vh, cl = vl, e = e_of(mt, h);
            if (mt + 1 < most_tiles) { vh = __ldg(frag + (mt + 1) * 64); vl = __ldg(frag + (mt + 1) * 64 + 32); }
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            mma_f16(c, cl.x, cl.y, cl.z, cl.w, e.x, e.y);
            mma_f16(c, ch.x, ch.y, ch.z, ch.w, e.z, e.w);
            mma_f16(c, ch.x, ch.y, ch.z, ch.w, e.x, e.y);
#pragma unroll
            for (int u = 0; u < 4; ++u) proj[u] += c[u];
        }
        const float vs = p.projected_scale[h];
        const float f0 = in0 ? vs * e_unit[2 * t][h] : 0.f, f1 = in1 ? vs * e_unit[2 * t + 1][h] : 0.f;
        proj[0] *= f0; proj[1] *= f1; proj[2] *= f0; proj[3] *= f1;
    } else {
        // ---- Psi: C[bin][row] of bin tile bt and NH heads; the node tiles in reach of the bins are consecutive
        constexpr int NH = 4;
        const int bt = warp & 3, h0 = (warp >> 2) * NH;
        const int2 reach = node_tiles_in_reach(bt, p.inv_wscale);
        const int most = min(most_tiles, reach.y);
        float psi[NH][4];
#pragma unroll
        for (int u = 0; u < NH; ++u) psi[u][0] = psi[u][1] = psi[u][2] = psi[u][3] = 0.f;
        const uint4 *frag = p.basis + bt * 64 + lane;
        int mt = reach.x;
        uint4 gh = make_uint4(0u, 0u, 0u, 0u), gl = gh;
        if (mt < most) { gh = __ldg(frag + mt * 256); gl = __ldg(frag + mt * 256 + 32); }
        for (; mt < most; ++mt) {
            const uint4 ch = gh, cl = gl;
            if (mt + 1 < most) { gh = __ldg(frag + (mt + 1) * 256); gl = __ldg(frag + (mt + 1) * 256 + 32); }
            // (a sum of its own per node tile, added in registers: the tensor pipe truncates what it adds to)
#pragma unroll
            for (int u = 0; u < NH; ++u) {
                const uint4 e = e_of(mt, h0 + u);
                float c[4] = {0.f, 0.f, 0.f, 0.f};
                mma_f16(c, cl.x, cl.y, cl.z, cl.w, e.x, e.y);
                mma_f16(c, ch.x, ch.y, ch.z, ch.w, e.z, e.w);
                mma_f16(c, ch.x, ch.y, ch.z, ch.w, e.x, e.y);
#pragma unroll
                for (int x = 0; x < 4; ++x) psi[u][x] += c[x];
            }
        }
        float4 wf[4][2];  // the projection's rows, on their way over the barriers
#pragma unroll
        for (int bb = 0; bb < 4; ++bb)
#pragma unroll
            for (int u = 0; u < 2; ++u)
                wf[bb][u] = __ldg(reinterpret_cast<const float4 *>(p.W + (h * HEAD_DIM + g + 8 * u) * 64 + bb * 16 + 4 * t));
        __syncthreads();  // (E has been read)
#pragma unroll
        for (int u = 0; u < NH; ++u) {
            const float s0 = in0 ? e_unit[2 * t][h0 + u] * (1.0f / PG_BASIS_SCALE) : 0.f, s1 = in1 ? e_unit[2 * t + 1][h0 + u] * (1.0f / PG_BASIS_SCALE) : 0.f;
            float *o = ps + (h0 + u) * 64 + bt * 16 + g;
            o[(2 * t) * PSI_LD] = psi[u][0] * s0; o[(2 * t + 1) * PSI_LD] = psi[u][1] * s1;
            o[(2 * t) * PSI_LD + 8] = psi[u][2] * s0; o[(2 * t + 1) * PSI_LD + 8] = psi[u][3] * s1;
        }
        __syncthreads();
        if (p.psi_row != nullptr)
            for (int at = tid; at < rows * 128; at += L::THREADS) {
                const int r = at >> 7, x = at & 127;
                if (row_tiles[r] > 0)
                    reinterpret_cast<float4 *>(p.psi_row + (a0 + i0 + r) * 512)[x] = *reinterpret_cast<const float4 *>(ps + r * PSI_LD + 4 * x);
            }
        // ---- projection: head h over the bins, in the order of the lane's pieces (by TF32 pairs 1.5 times a float32 product's error in
        // rows of few terms, and a tenth more than by three pieces on average)
#pragma unroll
        for (int bb = 0; bb < 4; ++bb) {
            const float4 w0 = wf[bb][0], w1 = wf[bb][1];
            const float4 x = *reinterpret_cast<const float4 *>(ps + g * PSI_LD + h * 64 + bb * 16 + 4 * t);
            const float bv[4] = {x.x, x.y, x.z, x.w};
            unsigned bh[4], bl[4], b3[4];
            split3_tf32(bv, bh, bl, b3);
            float pr[4];
            mma_exact(pr, {w0.x, w1.x, w0.y, w1.y}, {w0.z, w1.z, w0.w, w1.w}, bh, bl, b3);
#pragma unroll
            for (int u = 0; u < 4; ++u) proj[u] += pr[u];
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) val[u] += proj[u];
    float *o = p.out + (a0 + i0 + 2 * t) * (HEADS * HEAD_DIM) + h * HEAD_DIM + g;
    if (in0) { o[0] = val[0]; o[8] = val[2]; }
    if (in1) { o[128] = val[1]; o[136] = val[3]; }
    // An operand in pieces turns an infinity (of a value or of W) into a NaN: such rows are the row kernel's, whose products keep it.
    auto look = [&](bool in, int r, float sum) {
        if (!in || sum < INFINITY || atomicExch(odd + r, 1u) != 0u) return;
        p.leftover[atomicAdd(p.left_count, 1u)] = (int)(a0 + i0 + r);
        if (p.left != nullptr) p.left[a0 + i0 + r] = 1;
    };
    look(in0, 2 * t, fabsf(val[0]) + fabsf(val[2]));
    look(in1, 2 * t + 1, fabsf(val[1]) + fabsf(val[3]));
}

template <int TAIL, int STAGES>
int launch(const Args &p, long long blocks, cudaStream_t s)
{
    using L = Layout<TAIL, STAGES>;
    const size_t smem = L::bytes(p.max_atoms);
    auto kernel = pair_attn_kernel<TAIL, STAGES>;
    static thread_local bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured[dev & 63]) {
        const size_t most = L::bytes(PG_MAX_ATOMS);
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) {
            cudaGetLastError();
            return fail(CF_ERR_CUDA, "pair attention: %zu bytes of shared memory not available", most);
        }
        configured[dev & 63] = true;
    }
    launch_chained(kernel, dim3((unsigned)blocks), dim3(L::THREADS), smem, s, true, p);
    return launch_status("pair_attn_kernel");
}

// Three stages of copies where two blocks per SM leave room for them.
template <int TAIL>
int launch_fit(const Args &p, long long blocks, cudaStream_t s)
{
    constexpr size_t HALF_SM = 113 * 1024;
    return Layout<TAIL, 3>::bytes(p.max_atoms) <= HALF_SM ? launch<TAIL, 3>(p, blocks, s) : launch<TAIL, 2>(p, blocks, s);
}

}  // namespace

static int launch_pair_attn(const PairAttn &l, cudaStream_t s)
{
    if (l.N == 0) return CF_OK;
    Args p{};
    p.q = l.q; p.k = l.k; p.v = l.v; p.a = l.a; p.rvlen = l.rvlen; p.W = l.W; p.atom_start = l.atom_start; p.edge_start = l.edge_start;
    p.rule = l.rule; p.par = l.par; p.slots = l.grid.slots; p.tiles = l.grid.tiles; p.counters = l.grid.counters;
    p.left_count = l.grid.counters + 4 * (l.call + 1); p.leftover = l.leftover; p.left = l.left; p.basis = l.grid.basis;
    p.inv_wscale = l.wscale > 0 ? (float)(1.0 / (double)(float)l.wscale) : 1.0f;
    p.out = l.out; p.lse = l.lse; p.psi_row = l.psi_row; p.max_atoms = l.max_atoms; p.stats = row_stats_words();
    const long long blocks = l.N / PG_ROWS + l.B;
    if (l.K == 0) return launch_fit<PLAIN>(p, blocks, s);
    if (l.psi_row != nullptr || !l.projected) return launch_fit<KEEP_PSI>(p, blocks, s);
    p.projected = l.grid.projected + (size_t)l.call * HEADS * PG_TILES_BASIS * 64;
    p.projected_scale = l.grid.projected_scale + l.call * HEADS;
    return launch_fit<PROJECTED>(p, blocks, s);
}

int grid_attn_impl(const PairAttn &p, const float *pos_ij, const float *tvecs, const int64_t *batch, const int64_t *edges,
                   const int64_t *row_start, double cutoff_radius, int lattice_range, int minimum_range, cudaStream_t s)
{
    const int rc = launch_pair_attn(p, s);
    if (rc != CF_OK) return rc;
    unsigned *left = p.grid.counters + 4 * (p.call + 1);
    return launch_leftover_rows(p.q, p.k, p.v, p.a, pos_ij, tvecs, p.rvlen, batch, edges, row_start, p.N, p.E, p.max_atoms, p.dist_max,
                                p.wscale, p.W, cutoff_radius, lattice_range, minimum_range, p.out, p.logit, p.lse, p.psi_row, p.leftover, left,
                                left + 1, p.K, s);
}

namespace {
// What the entry points over a caller's grids share.
int grid_call(PairAttn &p, const char *who, const float *rvlen, const int64_t *atom_start, const int64_t *edge_start, int64_t N, int64_t B,
              int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale, double cutoff_radius, int lattice_range,
              int minimum_range, double a_widest, void *grids)
{
    CF_REQUIRE(N >= 0 && E >= 0 && B >= 0, CF_ERR_INVALID, "%s: negative size", who);
    CF_REQUIRE(K == 0 || K == 64, CF_ERR_UNSUPPORTED, "%s: K=%lld, only K in {0,64} is compiled", who, (long long)K);
    CF_REQUIRE(lattice_range >= 0 && lattice_range <= CF_MAX_RANGE && minimum_range >= 0, CF_ERR_RANGE, "%s: lattice_range %d outside [0,%d]", who,
               lattice_range, CF_MAX_RANGE);
    CF_REQUIRE(max_atoms >= 1 && max_atoms <= PG_MAX_ATOMS, CF_ERR_RANGE, "%s: max_atoms=%lld outside [1,%d]", who, (long long)max_atoms, PG_MAX_ATOMS);
    if (N == 0) return CF_OK;
    CF_REQUIRE(atom_start && edge_start && grids && (rvlen || cutoff_radius == 0), CF_ERR_INVALID, "%s: null pointer", who);
    CF_REQUIRE(pair_grid_fits(N, B, E, max_atoms, 64), CF_ERR_RANGE, "%s: %lld edges are more than grids are kept for", who, (long long)E);
    CF_REQUIRE(pair_grid_params(K, dist_max, wscale, (float)a_widest, weight_floor_log2(), p.par), CF_ERR_UNSUPPORTED,
               "%s: the nodes do not cover Gaussians of a_widest=%g (dist_max=%g, wscale=%g, floor 2^%g)", who, a_widest, dist_max, wscale,
               (double)weight_floor_log2());
    p.rvlen = cutoff_radius != 0.0 ? rvlen : nullptr;
    p.atom_start = atom_start; p.edge_start = edge_start; p.N = N; p.B = B; p.E = E; p.K = K; p.max_atoms = (int)max_atoms;
    p.rule = BoxRule{(float)cutoff_radius, lattice_range, minimum_range};
    p.dist_max = dist_max; p.wscale = wscale;
    p.grid = pair_grid_carve(grids, N, B, E, K);
    p.leftover = p.grid.leftover;
    return CF_OK;
}
// The kernels read rows in pieces of 16 bytes; a caller's tensors may lie anywhere
bool in_pieces(std::initializer_list<const void *> pointers)
{
    uintptr_t any = 0;
    for (const void *p : pointers) any |= (uintptr_t)p;
    return (any & 15) == 0;
}
// The rows that a forward marked, listed again for its backward
__global__ void list_left_kernel(const unsigned char *__restrict__ left, long long N, int *__restrict__ list, unsigned *__restrict__ count)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N && left[i] != 0) list[atomicAdd(count, 1u)] = (int)i;
}
}  // namespace
}  // namespace cf

extern "C" int64_t cf_pair_grid_bytes(int64_t N, int64_t B, int64_t E)
{
    if (N <= 0 || B <= 0 || E < 0) return 0;
    const size_t bytes = cf::pair_grid_bytes(N, B, E, 64);  // (for any K)
    return bytes <= cf::PG_MAX_BYTES ? (int64_t)bytes : 0;
}

extern "C" int cf_pair_grid_build(const float *pos_ij, const float *tvecs, const float *rvlen, const int64_t *atom_start,
                                  const int64_t *edge_start, int64_t N, int64_t B, int64_t E, int64_t max_atoms, int64_t K, double dist_max,
                                  double wscale, double cutoff_radius, int lattice_range, int minimum_range, double a_widest, void *grids,
                                  void *stream)
{
    using namespace cf;
    PairAttn p{};
    const int rc = grid_call(p, "cf_pair_grid_build", rvlen, atom_start, edge_start, N, B, E, K, max_atoms, dist_max, wscale, cutoff_radius,
                             lattice_range, minimum_range, a_widest, grids);
    if (rc != CF_OK || N == 0) return rc;
    CF_REQUIRE(pos_ij && tvecs, CF_ERR_INVALID, "cf_pair_grid_build: null pointer");
    return launch_pair_grid_build(p, pos_ij, tvecs, (float)a_widest, nullptr, 0, 0, as_stream(stream));
}

extern "C" int cf_infinite_attn_fwd_grid(const float *q, const float *k, const float *v, const float *a, const float *pos_ij,
                                         const float *tvecs, const float *rvlen, const int64_t *batch, const int64_t *edges,
                                         const int64_t *row_start, const int64_t *atom_start, const int64_t *edge_start, int64_t N, int64_t B,
                                         int64_t H, int64_t D, int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale,
                                         const float *W, double cutoff_radius, int lattice_range, int minimum_range, double a_widest,
                                         float *out, float *logit, float *lse, float *psi_row, uint8_t *left, void *grids, void *stream)
{
    using namespace cf;
    CF_REQUIRE(H == HEADS && D == HEAD_DIM, CF_ERR_UNSUPPORTED, "cf_infinite_attn_fwd_grid: H=%lld D=%lld, only H=8 D=16 is compiled",
               (long long)H, (long long)D);
    PairAttn p{};
    const int rc = grid_call(p, "cf_infinite_attn_fwd_grid", rvlen, atom_start, edge_start, N, B, E, K, max_atoms, dist_max, wscale,
                             cutoff_radius, lattice_range, minimum_range, a_widest, grids);
    if (rc != CF_OK || N == 0) return rc;
    CF_REQUIRE(q && k && v && a && pos_ij && tvecs && batch && edges && row_start && out && lse && (K == 0 || W), CF_ERR_INVALID,
               "cf_infinite_attn_fwd_grid: null pointer");
    CF_REQUIRE(in_pieces({q, k, v, out, lse, psi_row, W, grids}), CF_ERR_INVALID,
               "cf_infinite_attn_fwd_grid: q, k, v, W, out, lse, psi_row and grids must start on 16 bytes");
    p.q = q; p.k = k; p.v = v; p.a = a; p.W = W; p.out = out; p.lse = lse; p.psi_row = psi_row; p.logit = logit; p.left = left;
    p.call = PG_LAYERS - 1;  // (its counters are cleared here: any number of calls per build, in one stream's order)
    cudaStream_t s = as_stream(stream);
    if (cudaMemsetAsync(p.grid.counters + 4 * PG_LAYERS, 0, 4 * sizeof(unsigned), s) != cudaSuccess) return launch_status("cf_infinite_attn_fwd_grid");
    return grid_attn_impl(p, pos_ij, tvecs, batch, edges, row_start, cutoff_radius, lattice_range, minimum_range, s);
}

extern "C" int cf_infinite_attn_bwd_grid(const float *q, const float *k, const float *v, const float *a, const float *pos_ij,
                                         const float *tvecs, const float *rvlen, const int64_t *batch, const int64_t *edges,
                                         const int64_t *row_start, const int64_t *atom_start, const int64_t *edge_start, int64_t N, int64_t B,
                                         int64_t H, int64_t D, int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale,
                                         const float *W, double cutoff_radius, int lattice_range, int minimum_range, double a_widest,
                                         const float *logit, const float *lse, const uint8_t *left, const float *out, const float *gout,
                                         float *gq, float *gk, float *gv, float *ga, float *glogit, float *prob, void *grids, void *stream)
{
    using namespace cf;
    CF_REQUIRE(H == HEADS && D == HEAD_DIM, CF_ERR_UNSUPPORTED, "cf_infinite_attn_bwd_grid: H=%lld D=%lld, only H=8 D=16 is compiled",
               (long long)H, (long long)D);
    PairAttn p{};
    const int rc = grid_call(p, "cf_infinite_attn_bwd_grid", rvlen, atom_start, edge_start, N, B, E, K, max_atoms, dist_max, wscale,
                             cutoff_radius, lattice_range, minimum_range, a_widest, grids);
    if (rc != CF_OK || N == 0) return rc;
    CF_REQUIRE(q && k && v && a && pos_ij && tvecs && batch && edges && row_start && logit && lse && left && out && gout && gq && gk && gv &&
               ga && glogit && prob && (K == 0 || W), CF_ERR_INVALID, "cf_infinite_attn_bwd_grid: null pointer");
    CF_REQUIRE(in_pieces({q, k, v, out, gout, lse, W, gq, ga, glogit, prob, grids}), CF_ERR_INVALID,
               "cf_infinite_attn_bwd_grid: q, k, v, W, out, gout, lse, gq, ga, glogit, prob and grids must start on 16 bytes");
    p.q = q; p.k = k; p.v = v; p.a = a; p.W = W; p.out = const_cast<float *>(out); p.lse = const_cast<float *>(lse);
    p.logit = const_cast<float *>(logit); p.left = const_cast<uint8_t *>(left); p.gout = gout;
    p.gq = gq; p.gk = gk; p.gv = gv; p.ga = ga; p.glogit = glogit; p.prob = prob;
    p.call = PG_LAYERS - 1;
    cudaStream_t s = as_stream(stream);
    unsigned *count = p.grid.counters + 4 * PG_LAYERS;
    if (cudaMemsetAsync(count, 0, 4 * sizeof(unsigned), s) != cudaSuccess) return launch_status("cf_infinite_attn_bwd_grid");
    list_left_kernel<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(left, N, p.leftover, count);
    return grid_attn_bwd_impl(p, pos_ij, tvecs, batch, edges, row_start, s);
}
