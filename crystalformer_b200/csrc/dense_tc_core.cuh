// What the forward and backward dense kernels share (dense_tc.cu, dense_tc_bwd.cu): block roles, the weight stream, one
// 128 x 128 x 128 product, and the conversion of accumulator fragments into operands.
//
// A thread block carries a tile of 128 atom rows (or 64: half_tiles below) through its chain of products.  Warps 0-15 are the epilogue warps
// (thread = 4 rows x 8 columns of a 128 x 128 accumulator, in the layout of tmem_load_16x32: warp w covers rows
// 32 (w % 4) .., columns 32 (w / 4) ..; with eight warps an epilogue took 2 us instead of 1), one thread of warp 16
// issues the tensor instructions, one thread of warp 17 streams the weight images through a ring of three 32 KB stages.
// Operands: two 64 KB buffers in shared memory, each { h0, h1 } of two 64-deep k panels.  A product of two-piece operands is
// three fp16 products, h0 h1 + h1 h0 + h0 h0 (h1 h1 is below 2^-24 of a term), accumulated in fp32 in tensor memory.
// The tensor pipe drops what does not fit when it adds to an accumulator, always towards zero: half a unit of the sum per
// instruction.  So the small products come first, while the sum is 2^-11 of what it will be, and the eight instructions of
// h0 h0 last; and a sum of several products (feed-forward chunks, the three of the head's gradient) is made in registers,
// rounded to nearest, from an accumulator per product.  What is still lost is mostly a factor: the eight additions take
// 1.6e-7 of the result on average (regression on the operands of training steps, 1.2e-7 to 1.6e-7), of which the scales of
// the weights give 2^-23 back (not the embedding's: sums of one element per row lose nothing).
// Relative errors against 64 bits, float32 GEMMs on the same operands in brackets: 128-deep product 1.4e-7 (2.0e-7), 512-deep
// sum of chunks 2.5e-7 (3.5e-7); with the piece products in turn and the chunks in one accumulator 4.8e-7 and 1.8e-6; the
// TF32 + bfloat16 split of the warp-level version has 2^-20 per term.
#pragma once
#include "dense_tc.cuh"
#include "tc5.cuh"

#include "common.cuh"

namespace cf {
namespace tc5 {

constexpr int EPI_WARPS = 16, EPI_THREADS = 512, BLOCK_THREADS = 576;
constexpr int ISSUE_WARP = 16, STREAM_WARP = 17;
constexpr int STAGES = 3, STAGE_BYTES = 32768, OPERAND_BYTES = 65536;
constexpr int OFF_A0 = 0, OFF_A1 = OPERAND_BYTES, OFF_RING = 2 * OPERAND_BYTES, OFF_MISC = OFF_RING + STAGES * STAGE_BYTES;
// misc: barriers (16 x 8), tensor-memory address, give-up flag, then per-row floats
constexpr int OFF_ROW = OFF_MISC + 256;             // 5 x 128 floats: scales of loaded rows, row maxima of the column groups
constexpr int SMEM_BYTES = OFF_ROW + 5 * 512 + 64;  // (+ a word per epilogue warp)
static_assert(SMEM_BYTES <= 232448, "shared memory of one SM");
enum Barrier { B_FULL = 0, B_EMPTY = STAGES, B_D0 = 2 * STAGES, B_D1, B_DX, B_A0, B_A1, B_A1_FREE, B_DRAIN, B_PART, B_ROWS, B_GO };
constexpr float GIVEN_BACK = 1.0f + 0x1p-23f;  // see above; a factor of the weights' scales (powers of two: exact)
constexpr int D0 = 0, D1 = 128, DX = 256, DY = 384;  // accumulators (columns of tensor memory)

struct Shared {
    uint32_t base;              // shared address of the block's memory
    unsigned char *mem;
    volatile unsigned *gave_up;
    __device__ __forceinline__ uint32_t bar(int b) const { return base + OFF_MISC + 8u * (uint32_t)b; }
    __device__ __forceinline__ float *row_floats(int which) const { return reinterpret_cast<float *>(mem + OFF_ROW) + 128 * which; }
    __device__ __forceinline__ float *warp_floats() const { return reinterpret_cast<float *>(mem + OFF_ROW + 5 * 512); }
};

// The parities this thread waits for next.  An epilogue thread ignores a failed wait and carries on (all later waits
// then fail at once): the epilogue threads meet at named barriers and must stay together; what they compute after that
// is void, and the block reports it.
struct Phase {
    uint32_t bits = 0;
    __device__ __forceinline__ bool wait(const Shared &s, int b)
    {
        const bool ok = mbar_wait(s.bar(b), (bits >> b) & 1u, s.gave_up);
        bits ^= 1u << b;
        return ok;
    }
    __device__ __forceinline__ bool wait_cluster(const Shared &s, int b)  // arrivals from other blocks of the cluster
    {
        const bool ok = mbar_wait<true>(s.bar(b), (bits >> b) & 1u, s.gave_up);
        bits ^= 1u << b;
        return ok;
    }
};

// ---- weight stream (one thread) -------------------------------------------------------------------------------------
template <int STAGES>
struct Producer {
    int slot = 0;
    int requested = 0;   // stages asked for so far
    uint32_t phase = 1;  // the stages start out empty
    bool ok = true;
    __device__ __forceinline__ void stream(const Shared &s, const unsigned char *image, int first_block, int blocks, int pieces = 2)
    {
        const unsigned char *src = image + TC_HEADER_BYTES + (size_t)first_block * TC_BLOCK_BYTES;
        for (int i = 0; i < pieces * blocks && ok; ++i) {
            ok = mbar_wait(s.bar(B_EMPTY + slot), phase, s.gave_up);
            if (!ok) return;
            mbar_expect(s.bar(B_FULL + slot), STAGE_BYTES);
            bulk_load(s.base + OFF_RING + slot * STAGE_BYTES, src + (size_t)i * STAGE_BYTES, STAGE_BYTES, s.bar(B_FULL + slot));
            ++requested;
            if (++slot == STAGES) { slot = 0; phase ^= 1u; }
        }
    }
    // After a wait has run out: the copies still under way are waited for (with a limit of their own) before the block ends.
    __device__ __forceinline__ void drain(const Shared &s)
    {
        unsigned mine = 0u;
        for (int i = 0; i < STAGES; ++i)
            if (requested > i) mbar_wait(s.bar(B_FULL + i), (uint32_t)((requested - 1 - i) / STAGES) & 1u, &mine);
    }
};

// ---- tensor instructions (one thread) ---------------------------------------------------------------------------------
template <int STAGES>
struct Issuer {
    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    // D = A . B^T for the operand buffer at a_off and the next block of the stream, whose pieces come smallest first
    __device__ __forceinline__ void product(const Shared &s, uint32_t tmem, int d_col, int a_off, int pieces = 2)
    {
        constexpr uint32_t IDESC = instr_desc<128, 128, 0, false>();
        const uint64_t a0 = smem_desc(s.base + a_off, 16, 1024), a1 = smem_desc(s.base + a_off + 32768, 16, 1024);
        for (int left = pieces - 1; left >= 0 && ok; --left) {
            ok = mbar_wait(s.bar(B_FULL + slot), phase, s.gave_up);
            if (!ok) return;
            const uint64_t b = smem_desc(s.base + OFF_RING + slot * STAGE_BYTES, 16, 1024);
            // step ks: 16 k = 32 bytes = 2 units of the descriptor's address field, four to a panel of 16 KB = 1024 units
            auto at = [](int ks) { return (uint64_t)((ks >> 2) * 1024 + (ks & 3) * 2); };
            if (left == 0) {
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) mma_f16(tmem + d_col, a1 + at(ks), b + at(ks), IDESC, true);
            }
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) mma_f16(tmem + d_col, a0 + at(ks), b + at(ks), IDESC, left < pieces - 1 || ks > 0);
            mma_commit(s.bar(B_EMPTY + slot));
            if (++slot == STAGES) { slot = 0; phase ^= 1u; }
        }
    }
    // after a wait has run out: the instructions issued so far
    __device__ __forceinline__ void drain(const Shared &s)
    {
        unsigned mine = 0u;
        mma_commit(s.bar(B_DRAIN));
        mbar_wait(s.bar(B_DRAIN), 0, &mine);
    }
};

// ---- epilogue threads ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }

// this thread's place in a 128 x 128 accumulator: row(half, e) = row0 + 16 half + 8 e, columns col0 + 8 j + {0, 1}, j < 4.
// HALVES = 1: a tile of 64 rows, sixteen in each quarter of the accumulator (the rest is multiplied and never looked at: the tensor
// pipe is not what a tile waits for, and every epilogue is half as long).
template <int HALVES_>
struct PlaceOf {
    static constexpr int HALVES = HALVES_, ROWS = 64 * HALVES;
    int row0, col0, g, t, group;  // group: column group of 32
    int tile0;                    // row0 in the tile
    // the accumulator's row of a tile's row
    static __device__ __forceinline__ int accumulator_row(int row) { return HALVES == 2 ? row : (row >> 4) * 32 + (row & 15); }
    uint32_t tmem_off;            // lane and column offset of this warp's part (half 0)
    __device__ __forceinline__ PlaceOf()
    {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        g = lane >> 2; t = lane & 3; group = w >> 2;
        row0 = 32 * (w & 3) + g;
        tile0 = 16 * HALVES * (w & 3) + g;
        col0 = 32 * group + 2 * t;
        tmem_off = ((uint32_t)(32 * (w & 3)) << 16) + 32u * (uint32_t)group;
    }
    __device__ __forceinline__ uint32_t tmem(uint32_t base, int d_col, int half) const
    {
        return base + tmem_off + ((uint32_t)(16 * half) << 16) + (uint32_t)d_col;
    }
};
using Place = PlaceOf<2>;

// 16 values of `half` (rows scaled by s0 / s1) into an operand buffer
template <class P>
__device__ __forceinline__ void store_operand(unsigned char *buf, const P &pl, int half, const float (&v)[16], float s0, float s1)
{
    unsigned char *at = buf + (pl.group >> 1) * 16384 + (pl.row0 + 16 * half) * 128 + pl.t * 4;
    const int chunk0 = 4 * (pl.group & 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t h0, h1;
        unsigned char *c = at + (((chunk0 + j) ^ pl.g) << 4);
        split_pair(v[4 * j] * s0, v[4 * j + 1] * s0, h0, h1);
        *reinterpret_cast<uint32_t *>(c) = h0;
        *reinterpret_cast<uint32_t *>(c + 32768) = h1;
        split_pair(v[4 * j + 2] * s1, v[4 * j + 3] * s1, h0, h1);
        *reinterpret_cast<uint32_t *>(c + 1024) = h0;          // 8 rows further: the same swizzle phase
        *reinterpret_cast<uint32_t *>(c + 1024 + 32768) = h1;
    }
}

// sum += this thread's part of an accumulator whose product is known to be complete
template <class P>
__device__ __forceinline__ void add_accumulator(const P &pl, uint32_t tmem, int d_col, float (&sum)[2][16])
{
    fence_after();
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half) {
        float d[16];
        tmem_load_16x32(pl.tmem(tmem, d_col, half), d);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[half][i] += d[i];
    }
}

// largest magnitude of each of the thread's four rows over all 128 columns (the four column groups of the block);
// m[2 half + e].  Two barriers of the epilogue threads: the second one keeps a later call from overwriting maxima
// still being read.
template <class P>
__device__ __forceinline__ void row_maxima(const Shared &s, const P &pl, float (&m)[4])
{
#pragma unroll
    for (int i = 0; i < 2 * P::HALVES; ++i) {
        m[i] = fmaxf(m[i], __shfl_xor_sync(FULL, m[i], 1));
        m[i] = fmaxf(m[i], __shfl_xor_sync(FULL, m[i], 2));
    }
    if (pl.t == 0) {
        float *mine = s.row_floats(1 + pl.group);
#pragma unroll
        for (int i = 0; i < 2 * P::HALVES; ++i) mine[pl.row0 + 8 * i] = m[i];
    }
    epilogue_sync();
    const float *all = s.row_floats(1) + pl.row0;
#pragma unroll
    for (int i = 0; i < 2 * P::HALVES; ++i)
        m[i] = fmaxf(fmaxf(all[8 * i], all[128 + 8 * i]), fmaxf(all[256 + 8 * i], all[384 + 8 * i]));
    epilogue_sync();
}

// The block's rows as operand 0: scales from the largest magnitude of every row (xi: 1 / scale of the thread's rows).
template <class P>
__device__ __forceinline__ void publish_rows(const Shared &s, const P &pl, const float (&x)[2][16], float (&xi)[4])
{
    float m[4] = {0.f, 0.f, 0.f, 0.f}, xs[4];
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half)
#pragma unroll
        for (int i = 0; i < 16; ++i) m[2 * half + ((i >> 1) & 1)] = fmaxf(m[2 * half + ((i >> 1) & 1)], fabsf(x[half][i]));
    row_maxima(s, pl, m);
#pragma unroll
    for (int i = 0; i < 4; ++i) xs[i] = power_of_two(m[i], xi[i]);
#pragma unroll
    for (int half = 0; half < P::HALVES; ++half) store_operand(s.mem + OFF_A0, pl, half, x[half], xs[2 * half], xs[2 * half + 1]);
    fence_async_smem();
    fence_before();
    mbar_arrive(s.bar(B_A0));
}

// this thread's eight values of a per-column constant (read before the wait for the product that needs them)
template <class P>
__device__ __forceinline__ void load_columns(const float *src, const P &pl, float2 (&b)[4])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float2 *>(src + pl.col0 + 8 * j);
}

// two columns of a row-major (N, ld) array at this thread's fragment positions of `half`, zero beyond row N
template <class P>
__device__ __forceinline__ void load_rows(const float *src, int ld, long long row_base, long long N, const P &pl, int half, float (&v)[16])
{
    const long long r0 = row_base + pl.tile0 + 16 * half, r1 = r0 + 8;
    const float *p0 = src + r0 * ld + pl.col0, *p1 = src + r1 * ld + pl.col0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 a = r0 < N ? *reinterpret_cast<const float2 *>(p0 + 8 * j) : make_float2(0.f, 0.f);
        const float2 b = r1 < N ? *reinterpret_cast<const float2 *>(p1 + 8 * j) : make_float2(0.f, 0.f);
        v[4 * j] = a.x; v[4 * j + 1] = a.y; v[4 * j + 2] = b.x; v[4 * j + 3] = b.y;
    }
}
template <class P>
__device__ __forceinline__ void store_rows(float *dst, int ld, long long row_base, long long N, const P &pl, int half, const float (&v)[16])
{
    const long long r0 = row_base + pl.tile0 + 16 * half, r1 = r0 + 8;
    float *p0 = dst + r0 * ld + pl.col0, *p1 = dst + r1 * ld + pl.col0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (r0 < N) *reinterpret_cast<float2 *>(p0 + 8 * j) = make_float2(v[4 * j], v[4 * j + 1]);
        if (r1 < N) *reinterpret_cast<float2 *>(p1 + 8 * j) = make_float2(v[4 * j + 2], v[4 * j + 3]);
    }
}

// Loads a tile of rows as an operand: warp w takes eight (four) rows from 8 w (4 w) on, lane l the columns 4 l .. 4 l + 3 (fetch(row,
// lane) returns them); the row's scale comes from its own largest magnitude, 1 / scale goes to row_floats(0).
template <class P = Place, class Fetch>
__device__ __forceinline__ void load_operand(const Shared &s, unsigned char *buf, Fetch &&fetch)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *inv_out = s.row_floats(0);
    constexpr int EACH = 4 * P::HALVES;
    float4 v[EACH];
    float m[8] = {};
#pragma unroll
    for (int u = 0; u < EACH; ++u) v[u] = fetch(EACH * w + u, lane);
#pragma unroll
    for (int u = 0; u < EACH; ++u) m[u] = fmaxf(fmaxf(fabsf(v[u].x), fabsf(v[u].y)), fmaxf(fabsf(v[u].z), fabsf(v[u].w)));
    const float row_max = warp_max_of_8(m, lane);  // of row lane / 4
#pragma unroll
    for (int u = 0; u < EACH; ++u) {
        const int row = P::accumulator_row(EACH * w + u);
        float inv;
        const float sc = power_of_two(__shfl_sync(FULL, row_max, 4 * u), inv);
        if (lane == 0) inv_out[row] = inv;
        uint2 h0, h1;
        split_pair(v[u].x * sc, v[u].y * sc, h0.x, h1.x);
        split_pair(v[u].z * sc, v[u].w * sc, h0.y, h1.y);
        unsigned char *c = buf + (lane >> 4) * 16384 + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + (lane & 1) * 8;
        *reinterpret_cast<uint2 *>(c) = h0;
        *reinterpret_cast<uint2 *>(c + 32768) = h1;
    }
}

// ---- a tile shared by four blocks ---------------------------------------------------------------------------------------
// A boundary is a chain of twelve products per tile, about a microsecond each on one SM's tensor pipe; with few tiles most
// SMs have none.  A cluster of four blocks then takes a tile: block r multiplies hidden chunk r and head matrix r, products
// that precede them are done by all four.  Where the chunks meet in one sum, every block sends its share of rows
// 32 o .. 32 o + 31 to block o (slot r of operand buffer 1, which these blocks do not use otherwise); block o adds the four
// in rank order, finishes its 32 rows and, where they are the next operand, writes them into operand buffer 0 of every
// block that needs them.  Both transfers are bulk copies between the blocks' shared
// memories, from a staging place of the sender (shares: its operand buffer 0; finished rows: the third stage of the weight
// ring, which these blocks do without) with the bytes counted on the receiver's barrier, B_PART and B_ROWS: 3.5 us for the
// shares and 2.2 for the rows, against 3.9 and 2.7 with plain stores to the other blocks (48 KB leave every block: about 17
// bytes per ns, what an SM's link to the others in its cluster gives).  Rows may overwrite a
// receiver's operand buffer 0 once its own shares have left it: every block tells the others when it has received all of
// its shares (B_GO).
constexpr int SPLIT = 4, SPLIT_STAGES = STAGES - 1;
constexpr int OFF_STAGING = OFF_RING + SPLIT_STAGES * STAGE_BYTES;
constexpr int OFF_OWN = OFF_STAGING + 16384;     // the forward's residual of the rows that this block finishes
constexpr int OFF_STAGED_INV = OFF_ROW + 4 * 512;  // (row floats 4)
constexpr int SHARE_BYTES = 16384, ROWS_BYTES = 16384 + 128;

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t at_rank(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync()  // every thread of the four blocks
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void arrive_at(uint32_t bar_of_rank)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_of_rank) : "memory");
}
// shared memory of this block -> shared memory of another, the bytes counted on a barrier there
__device__ __forceinline__ void bulk_send(uint32_t dst_of_rank, uint32_t src, uint32_t bytes, uint32_t bar_of_rank)
{
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_of_rank),
                 "r"(src), "r"(bytes), "r"(bar_of_rank)
                 : "memory");
}
// (one thread of the receiver, once per transfer; the bytes may come first)
__device__ __forceinline__ void expect_shares(const Shared &s) { mbar_expect(s.bar(B_PART), SPLIT * SHARE_BYTES); }
__device__ __forceinline__ void expect_rows(const Shared &s) { mbar_expect(s.bar(B_ROWS), SPLIT * ROWS_BYTES); }

// 32 rows of 128 floats as they are staged: a row is 512 bytes, its 32-byte pieces swizzled by the row so that a warp's
// stores meet no bank twice.  One half (16 values) of this thread's part, and four columns of a row.
__device__ __forceinline__ void stage_rows(unsigned char *share, const Place &pl, int half, const float (&v)[16])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        unsigned char *at = share + (pl.g + 16 * half) * 512 + (((4 * pl.group + j) ^ pl.g) << 5) + pl.t * 8;
        *reinterpret_cast<float2 *>(at) = make_float2(v[4 * j], v[4 * j + 1]);
        *reinterpret_cast<float2 *>(at + 8 * 512) = make_float2(v[4 * j + 2], v[4 * j + 3]);
    }
}
__device__ __forceinline__ const float4 &staged_row(const unsigned char *share, int row, int lane)
{
    return *reinterpret_cast<const float4 *>(share + row * 512 + (((lane >> 1) ^ (row & 7)) << 5) + (lane & 1) * 16);
}
// A half of this thread's part of the share, for the block that finishes these rows.
__device__ __forceinline__ void stage_share(const Shared &s, const Place &pl, int half, const float (&v)[16])
{
    stage_rows(s.mem + OFF_A0 + ((threadIdx.x >> 5) & 3) * SHARE_BYTES, pl, half, v);
}
// The four warps that staged a share meet, and one thread sends it.
__device__ __forceinline__ void send_share(const Shared &s, uint32_t rank)
{
    const uint32_t to = (threadIdx.x >> 5) & 3u;
    fence_async_smem();
    fence_before();
    asm volatile("bar.sync %0, 128;" ::"r"(2u + to) : "memory");
    if ((threadIdx.x & 31) == 0 && (threadIdx.x >> 7) == 0)
        bulk_send(at_rank(s.base + OFF_A1 + rank * SHARE_BYTES, to), s.base + OFF_A0 + to * SHARE_BYTES, SHARE_BYTES, at_rank(s.bar(B_PART), to));
}
// The sums of this block's rows, once the four shares are here: row 2 w + u of its 32, columns 4 l .. 4 l + 3.
__device__ __forceinline__ void collect_shares(const Shared &s, Phase &ph, float4 (&v)[2])
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    ph.wait_cluster(s, B_PART);
    if (w == 0 && lane < SPLIT) arrive_at(at_rank(s.bar(B_GO), (uint32_t)lane));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int row = 2 * w + u;
        float4 a = staged_row(s.mem + OFF_A1, row, lane);
#pragma unroll
        for (int slot = 1; slot < SPLIT; ++slot) {
            const float4 b = staged_row(s.mem + OFF_A1 + slot * SHARE_BYTES, row, lane);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
        v[u] = a;
    }
}
// The block's finished rows as operand 0 (and 1 / scale as row floats `which`) of the first `receivers` blocks.
__device__ __forceinline__ void spread_rows(const Shared &s, Phase &ph, uint32_t rank, const float4 (&v)[2], int receivers, int which)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float m[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) m[u] = fmaxf(fmaxf(fabsf(v[u].x), fabsf(v[u].y)), fmaxf(fabsf(v[u].z), fabsf(v[u].w)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < 2; ++u) m[u] = fmaxf(m[u], __shfl_xor_sync(FULL, m[u], o));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int row = 2 * w + u;
        float inv;
        const float sc = power_of_two(m[u], inv);
        uint2 h0, h1;
        split_pair(v[u].x * sc, v[u].y * sc, h0.x, h1.x);
        split_pair(v[u].z * sc, v[u].w * sc, h0.y, h1.y);
        // staged by (k panel, piece): 32 rows x 128 bytes each, as the operand has them
        unsigned char *at = s.mem + OFF_STAGING + (lane >> 4) * 8192 + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + (lane & 1) * 8;
        *reinterpret_cast<uint2 *>(at) = h0;
        *reinterpret_cast<uint2 *>(at + 4096) = h1;
        if (lane == 0) *reinterpret_cast<float *>(s.mem + OFF_STAGED_INV + row * 4) = inv;
    }
    fence_async_smem();
    epilogue_sync();
    if (w == 0) {
        const int to = lane >> 2, part = lane & 3;  // (k panel, piece)
        ph.wait_cluster(s, B_GO);
        if (to < receivers) {
            const uint32_t bar = at_rank(s.bar(B_ROWS), (uint32_t)to), from = s.base + OFF_STAGING + part * 4096;
            bulk_send(at_rank(s.base + OFF_A0 + (part >> 1) * 16384 + (part & 1) * 32768 + rank * 4096u, (uint32_t)to), from, 4096, bar);
            if (part == 0)
                bulk_send(at_rank(s.base + OFF_ROW + (uint32_t)(which * 512) + rank * 128u, (uint32_t)to), s.base + OFF_STAGED_INV, 128, bar);
        }
    }
}
// positions of a chunk's two blocks in the interleaved order of an image (first the block that makes the hidden units)
__device__ __forceinline__ int first_of_chunk(int c) { return c < 2 ? c : 2 * c - 1; }
__device__ __forceinline__ int second_of_chunk(int c, int chunks) { return min(c + 2, chunks) + c; }

// ---- block set-up and end -----------------------------------------------------------------------------------------------
__device__ __forceinline__ Shared block_begin(unsigned char *mem, uint32_t &tmem)
{
    Shared s;
    s.mem = mem;
    s.base = smem_u32(mem);
    s.gave_up = reinterpret_cast<volatile unsigned *>(mem + OFF_MISC + 192);
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(s.bar(B_FULL + i), 1); mbar_init(s.bar(B_EMPTY + i), 1); }
        mbar_init(s.bar(B_D0), 1); mbar_init(s.bar(B_D1), 1); mbar_init(s.bar(B_DX), 1);
        mbar_init(s.bar(B_A0), EPI_THREADS); mbar_init(s.bar(B_A1), EPI_THREADS); mbar_init(s.bar(B_A1_FREE), 1);
        mbar_init(s.bar(B_DRAIN), 1);
        mbar_init(s.bar(B_PART), 1); mbar_init(s.bar(B_ROWS), 1); mbar_init(s.bar(B_GO), SPLIT);
        *s.gave_up = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if ((threadIdx.x >> 5) == ISSUE_WARP) tmem_alloc<512>(s.base + OFF_MISC + 200);
    fence_before();
    __syncthreads();
    fence_after();
    tmem = *reinterpret_cast<volatile uint32_t *>(mem + OFF_MISC + 200);
    return s;
}
__device__ __forceinline__ void block_end(const Shared &s, uint32_t tmem, unsigned *status)
{
    fence_before();
    __syncthreads();
    fence_after();
    if ((threadIdx.x >> 5) == ISSUE_WARP) tmem_free<512>(tmem);
    if (threadIdx.x == 0) report_waits(s.gave_up, status);
}

// ---- host side ------------------------------------------------------------------------------------------------------------
// The rule: a cluster per tile while all clusters fit at once (with a second wave, 41 tiles: 52 us against 39 with a block
// per tile, forward; 56 against 41 backward), one chunk per block at most, and not where the caller asked for the least SM
// time (dense_tile_rows 32: batches on several streams; four blocks of 20 us take more of the chip than one of 30, and a
// stream of 128-crystal batches on four streams 3.52 ms instead of 3.31).
inline bool split_tiles(long long tiles, int ff, int clusters)
{
    return ff <= 128 * SPLIT && tiles <= clusters && dense_tile_rows_choice() != 32;
}

// Otherwise tiles of 64 rows while there is an SM for each (and SM time is not what counts): every epilogue of the chain is half as
// long, and the products, which are not what it waits for, take as long as before.  Median of a network's boundaries with tiles
// of 128 and of 64: 4,881 rows 31 and 24 us (inference), 39 and 30 (training, forward), 48 and 33 (backward); 9,301 rows 32 and 32, 49
// and 34, 52 and 35.  Beyond 64 rows per SM a second tile would follow: 35 us twice against 50.
inline bool half_tiles(long long rows) { return (rows + 63) / 64 <= sm_count() && dense_tile_rows_choice() != 32; }

struct DenseLaunch {  // per thread: what a device's set-up of the kernels gave
    int clusters_of[64] = {};  // clusters that fit at once; 0: not set up yet
    int device = 0;
    int configure(const void *alone, const void *half, const void *split, const char *what)
    {
        int dev = 0;
        cudaGetDevice(&dev);
        device = dev & 63;
        if (clusters_of[device] > 0) return CF_OK;
        if (cudaFuncSetAttribute(alone, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
            cudaFuncSetAttribute(half, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
            cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) {
            cudaGetLastError();
            return fail(CF_ERR_CUDA, "%s: %d bytes of shared memory not available", what, SMEM_BYTES);
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(SPLIT); cfg.blockDim = dim3(BLOCK_THREADS); cfg.dynamicSmemBytes = SMEM_BYTES;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = SPLIT; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, split, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = sm_count() / SPLIT;
        }
        clusters_of[device] = n;
        return CF_OK;
    }
    int clusters() const { return clusters_of[device]; }
};

}  // namespace tc5
}  // namespace cf
