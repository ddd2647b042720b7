// What the attention kernels over pair grids share: one key tile's vectors in flight, functions at the nodes as operands.
#pragma once
#include "lattice_core.cuh"
#include "mma_frag.cuh"
#include "pair_grid.cuh"

namespace cf {

constexpr int PA_KEYS = 16;                        // keys per tile
constexpr int PA_STEP = 3;                         // node tiles per copy
constexpr float PA_W_SCALE = 32768.0f;             // weights and Gaussians at the nodes, as half pairs: exact to 2^-22 down to 2^-17
constexpr float PA_MAX_LAG = 16.0f;                // rows whose largest logit exceeds their own by more bits are left over
constexpr float PA_USUAL_LAG = 4.0f;               // ... and by which the nodes in reach are chosen before the logits are known

// Tables of a row, in the order in which a lane takes its operands of a product over the keys: per key tile 32 lanes (head g, t) x
// keys 2t, 2t + 1, 2t + 8, 2t + 9; rows 16 bytes beyond a multiple of 128 apart.
__host__ __device__ inline int pa_row_words(int max_atoms) { return ((max_atoms + PA_KEYS - 1) / PA_KEYS) * 128 + 4; }
// ... and the place of key j (0 ... 7; + 2 words: key j + 8) of head h
__device__ __forceinline__ int pa_key_word(int h, int j) { return h * 16 + (j >> 1) * 4 + (j & 1); }

// The rows' sums S lie in the order in which a product over the nodes leaves them: per key tile the lanes' four values (keys g,
// g + 8; heads 2t, 2t + 1), in an order of the lanes that meets no bank twice either way.
__device__ __forceinline__ int pa_sum_slot(int g, int t) { return t * 8 + ((g + 2 * t) & 7); }

// The vectors of a row on their way through a warp's ring of stages: a step is a key tile's values at up to STEP node tiles,
// key rows 16 bytes longer than their data (an odd number of 16 bytes: the eight rows of an ldmatrix take eight bank groups).
// (Offsets within a crystal and variant fit 32 bits: 51,360 pairs of 768 bytes at most.)
template <int STAGES>
struct KeyRing {
    static constexpr int KEY_LD = PA_STEP * 64 + 16, STAGE = PA_KEYS * KEY_LD, BYTES = STAGES * STAGE;
    const unsigned char *base, *k0, *k1;  // vectors of the crystal and variant, of the lane's keys
    int i, n, slot_bytes, key_tiles, lane_key, lane_byte;
    int ft, fs, tiles, put, got;          // next step to fetch (key tile, first node tile of the pass's so many), stages
    int pass, remaining;                  // node tiles of a pass; those of the passes to come
    unsigned ring, dst, plain, trans;     // the lane's place in a stage: copies, ldmatrix, ldmatrix transposed
    __device__ __forceinline__ void init(unsigned ring_, int i_, int n_, int slot_bytes_, int lane)
    {
        ring = ring_; i = i_; n = n_; slot_bytes = slot_bytes_;
        key_tiles = (n + PA_KEYS - 1) / PA_KEYS;
        lane_key = lane >> 2;
        lane_byte = (lane & 3) * 16;
        dst = ring + lane_key * KEY_LD + lane_byte;
        plain = ring + ((lane & 7) + 8 * ((lane >> 3) & 1)) * KEY_LD + (lane >> 4) * 16;
        trans = ring + ((lane & 7) + 8 * (lane >> 4)) * KEY_LD + ((lane >> 3) & 1) * 16;
    }
    __device__ __forceinline__ const unsigned char *at(int j) const
    {
        j = min(j, n - 1);
        const int lo = min(i, j), hi = max(i, j);
        return base + (unsigned)(((lo * (2 * n - 1 - lo)) >> 1) + hi) * (unsigned)slot_bytes;
    }
    __device__ __forceinline__ void fetch()
    {
        if (ft < key_tiles) {
            if (fs == 0) {
                const int j = ft * PA_KEYS + lane_key;
                k0 = at(j);
                k1 = at(j + 8);
            }
            const unsigned d = dst + put * STAGE;
            const unsigned char *s0 = k0 + fs * 64, *s1 = k1 + fs * 64;
#pragma unroll
            for (int u = 0; u < PA_STEP; ++u)
                if (u == 0 || fs + u < tiles) {
                    copy16_async(d + u * 64, s0 + u * 64);
                    copy16_async(d + 8 * KEY_LD + u * 64, s1 + u * 64);
                }
            put = put + 1 == STAGES ? 0 : put + 1;
            fs += PA_STEP;
            if (fs >= tiles) {
                fs = 0;
                if (++ft == key_tiles && remaining > 0) {  // on to the next pass over the keys
                    base += pass * 64;
                    tiles = min(pass, remaining);
                    remaining -= tiles;
                    ft = 0;
                }
            }
        }
        copy_commit();
    }
    // `total` node tiles of a variant's vectors from `first_tile`, in passes over the keys of up to `pass` tiles
    __device__ __forceinline__ void start(const unsigned char *vectors, int first_tile, int total, int pass_)
    {
        base = vectors + first_tile * 64 + lane_byte;
        pass = pass_;
        tiles = min(pass, total);
        remaining = total - tiles;
        ft = fs = put = got = 0;
#pragma unroll
        for (int u = 0; u < STAGES - 1; ++u) fetch();
    }
    // the oldest step's offset; every take is followed by a done
    __device__ __forceinline__ unsigned take()
    {
        fetch();
        copy_wait<STAGES - 1>();
        __syncwarp();
        const unsigned a = got * STAGE;
        got = got + 1 == STAGES ? 0 : got + 1;
        return a;
    }
    __device__ __forceinline__ void done() const { __syncwarp(); }
};

// What a row's heads are: the lanes of head g hold its Gaussian and its variant of the crystal's boxes.
struct RowHeads {
    float a2h2;      // exp(a d^2) = 2^(a2h2 m^2) at m nodes from zero, head g
    int variant;     // -1: the rule's box is none of the crystal's
    bool narrow;     // beyond what the nodes resolve, or not a Gaussian
};
__device__ __forceinline__ RowHeads row_heads(float a, const BoxRule &rule, const float *rvlen3, int4 info, const PairGridParams &par)
{
    RowHeads r;
    r.a2h2 = a * par.gauss;
    r.narrow = !(a < 0.0f && a >= par.a_least);
    if (info.y == (1 | (1 << 8) | (1 << 16) | PG_ALL_BOXES) && a <= par.a_widest) {  // one box whatever the width
        r.variant = 0;
        return r;
    }
    const int pk = packed_box(rule, a, rvlen3);
    const int d1 = box_r1(pk) - box_r1(info.x), d2 = box_r2(pk) - box_r2(info.x), d3 = box_r3(pk) - box_r3(info.x);
    const int e1 = info.y & 0xff, e2 = (info.y >> 8) & 0xff, e3 = (info.y >> 16) & 0xff;
    const bool there = d1 >= 0 && d1 < e1 && d2 >= 0 && d2 < e2 && d3 >= 0 && d3 < e3;
    r.variant = there ? d1 + e1 * (d2 + e2 * d3) : -1;
    return r;
}
// Node tiles in reach of the row's heads: the atom's own image is in every box at distance zero, so a head's sum is at least
// 2^-lag of its largest weight (lag: by how many bits the row's largest logit exceeds its own), and nodes beyond are below the
// floor against that.  More than par.tiles: not all are there.
__device__ __forceinline__ int row_tiles_of(const RowHeads &r, float lag, const PairGridParams &par)
{
    const float reach = sqrtf((lag - par.floor_log2) / -r.a2h2);
    const bool there = reach <= (float)(par.tiles * PG_TILE - PG_POINTS);
    // (a reduction instruction: what depends on its result is known to be the same in all lanes)
    return __reduce_max_sync(FULL, there ? min(((int)reach + PG_POINTS) / PG_TILE + 1, par.tiles) : par.tiles + 1);
}
// The largest logit of head g, in bits; row: the row's logits
__device__ __forceinline__ float row_top(const float *row, int key_tiles, int lane)
{
    float top = -INFINITY;
    for (int T = 0; T < key_tiles; ++T) {
        const float4 u = reinterpret_cast<const float4 *>(row)[T * 32 + lane];
        top = fmaxf(fmaxf(top, fmaxf(u.x, u.y)), fmaxf(u.z, u.w));
    }
    top = fmaxf(top, __shfl_xor_sync(FULL, top, 1));
    return fmaxf(top, __shfl_xor_sync(FULL, top, 2));
}

// Gaussians x = 2^(a2h2 m^2) of a lane at nodes m0, m0 + 1 (m counted from the node at distance zero)
__device__ __forceinline__ float2 gauss2(float a2h2, float m0)
{
    const float2 f = make_float2(m0, m0 + 1.0f);
    const float2 e = mul2(mul2(f, f), make_float2(a2h2, a2h2));
    return make_float2(ex2(e.x), ex2(e.y));
}

// The row's weights 2^(logit - top) in place of the logits, as operands of a product over the keys (B: keys x heads): values of
// keys 2t, 2t + 1 | 2t + 8, 2t + 9 and their remainders.  Keys beyond the last have the logit -inf: weight 0.
__device__ __forceinline__ void weights_in_place(float *row, int key_tiles, float top, int lane)
{
    for (int T = 0; T < key_tiles; ++T) {
        float4 *at = reinterpret_cast<float4 *>(row) + T * 32 + lane;
        const float4 u = *at;
        const float2 x = mul2(make_float2(ex2(u.x - top), ex2(u.y - top)), make_float2(PA_W_SCALE, PA_W_SCALE));
        const float2 y = mul2(make_float2(ex2(u.z - top), ex2(u.w - top)), make_float2(PA_W_SCALE, PA_W_SCALE));
        uint4 w;
        split_f16(x.x, x.y, w.x, w.z);
        split_f16(y.x, y.y, w.y, w.w);
        *reinterpret_cast<uint4 *>(at) = w;
    }
}
// ... back as numbers (scaled)
__device__ __forceinline__ float4 weights_of(uint4 w)
{
    const float2 a = add2(half2_of(w.x), half2_of(w.z)), b = add2(half2_of(w.y), half2_of(w.w));
    return make_float4(a.x, a.y, b.x, b.y);
}

// Products of eight rows (the lane's row g: row16) and their crystal's keys in one head, into the rows' tables, by TF32 pairs:
// C[key][row]; the contraction runs over the head's sixteen channels in the order in which a lane's 16-byte pieces hold them.
// Key tiles first, first + stride, ...
struct HeadOperands {  // the lane's pieces of its row and of the first two keys
    float4 row, k0, k1;
};
__device__ __forceinline__ HeadOperands head_operands(const float *__restrict__ row16, const float *__restrict__ keys, int n, int first, int lane)
{
    const int g = lane >> 2, t = lane & 3;
    const float4 *kp = reinterpret_cast<const float4 *>(keys) + t;
    HeadOperands o;
    o.row = *reinterpret_cast<const float4 *>(row16 + 4 * t);
    o.k0 = kp[min(first * PA_KEYS + g, n - 1) * (HEADS * HEAD_DIM / 4)];
    o.k1 = kp[min(first * PA_KEYS + g + 8, n - 1) * (HEADS * HEAD_DIM / 4)];
    return o;
}
template <bool SUM_ORDER>
__device__ __forceinline__ void head_products(const HeadOperands &op, const float *__restrict__ keys, int n, int head, int first, int stride,
                                              int key_tiles, float scale, float pad, float *table, int row_words, int lane)
{
    const int g = lane >> 2, t = lane & 3;
    const float bv[4] = {op.row.x * scale, op.row.y * scale, op.row.z * scale, op.row.w * scale};
    unsigned bh[4], bl[4], b3[4];
    split3_tf32(bv, bh, bl, b3);
    const float4 *kp = reinterpret_cast<const float4 *>(keys) + t;
    auto key = [&](int j) { return kp[min(j, n - 1) * (HEADS * HEAD_DIM / 4)]; };
    float4 k0 = op.k0, k1 = op.k1;
    const int slot = SUM_ORDER ? pa_sum_slot(g, head >> 1) * 4 + (head & 1) : pa_key_word(head, g);  // (SUM_ORDER: that of the sums S)
    float *o = table + 2 * t * row_words + first * 128 + slot;
    for (int T = first; T < key_tiles; T += stride, o += stride * 128) {
        const float4 a0 = k0, a1 = k1;
        const int j = T * PA_KEYS + g;
        if (T + stride < key_tiles) { k0 = key(j + stride * PA_KEYS); k1 = key(j + stride * PA_KEYS + 8); }
        // (a logit's error goes into the weight as it is, times the logit: with two pieces the rows of 24 crystals of up to 30 atoms
        // are 1.63e-7 from 64 bits, with three 1.48e-7, float32 sums 1.48e-7)
        float c[4];
        mma_exact(c, {a0.x, a1.x, a0.y, a1.y}, {a0.z, a1.z, a0.w, a1.w}, bh, bl, b3);
        o[0] = j < n ? c[0] : pad;
        o[row_words] = j < n ? c[1] : pad;
        o[2] = j + 8 < n ? c[2] : pad;
        o[row_words + 2] = j + 8 < n ? c[3] : pad;
    }
}

// The node tiles { first, end } that the basis functions of bin tile bt reach (6.6 standard deviations: 2^-31 beyond)
__device__ __forceinline__ int2 node_tiles_in_reach(int bt, float inv_wscale)
{
    const float lo = ((float)(bt * 16 + 1) * inv_wscale - 6.6f) * 3.0f + (float)PG_BELOW, hi = ((float)(bt * 16 + 16) * inv_wscale + 6.6f) * 3.0f + (float)PG_BELOW;
    return make_int2(max((int)floorf(lo * (1.0f / PG_TILE)), 0), min((int)floorf(hi * (1.0f / PG_TILE)) + 1, PG_TILES_BASIS));
}

}  // namespace cf
