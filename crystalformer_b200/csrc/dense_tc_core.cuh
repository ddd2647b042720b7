// What the forward and backward dense kernels share (dense_tc.cu, dense_tc_bwd.cu): block roles, the weight stream, one
// 128 x 128 x 128 product, and the conversion of accumulator fragments into operands.
//
// A thread block carries a tile of 128 atom rows (or 64 or 32: tile_rows below) through its chain of products.  Warps 0-15 are the epilogue warps
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
enum Barrier { B_FULL = 0, B_EMPTY = STAGES, B_D0 = 2 * STAGES, B_D1, B_DX, B_A0, B_A1, B_A1_FREE, B_DRAIN };
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
};

// ---- weight stream (one thread) -------------------------------------------------------------------------------------
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
// Tiles of 128, 64 and 32 rows: of a quarter of the accumulator the first 32, 16 and 8 rows are the tile's (the rest is multiplied and
// never looked at: the tensor pipe is not what a tile waits for, and every epilogue is half or a quarter as long).
template <int ROWS_>
struct PlaceOf {
    static constexpr int ROWS = ROWS_, HALVES = ROWS == 128 ? 2 : 1, PAIRS = ROWS == 32 ? 1 : 2;  // rows of a thread: (half, e < PAIRS)
    static constexpr int EACH = ROWS / 16;  // rows of a warp that loads or finishes whole rows
    int row0, col0, g, t, group;  // group: column group of 32
    int tile0;                    // row0 in the tile
    uint32_t tmem_off;            // lane and column offset of this warp's part (half 0)
    // the accumulator's row of a tile's row
    static __device__ __forceinline__ int accumulator_row(int row) { return row / (ROWS / 4) * 32 + row % (ROWS / 4); }
    __device__ __forceinline__ PlaceOf()
    {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        g = lane >> 2; t = lane & 3; group = w >> 2;
        row0 = 32 * (w & 3) + g;
        tile0 = ROWS / 4 * (w & 3) + g;
        col0 = 32 * group + 2 * t;
        tmem_off = ((uint32_t)(32 * (w & 3)) << 16) + 32u * (uint32_t)group;
    }
    __device__ __forceinline__ uint32_t tmem(uint32_t base, int d_col, int half) const
    {
        return base + tmem_off + ((uint32_t)(16 * half) << 16) + (uint32_t)d_col;
    }
};

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
        if (P::PAIRS == 1) continue;
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
    for (int i = 0; i < P::HALVES * P::PAIRS; ++i) {
        m[i] = fmaxf(m[i], __shfl_xor_sync(FULL, m[i], 1));
        m[i] = fmaxf(m[i], __shfl_xor_sync(FULL, m[i], 2));
    }
    if (pl.t == 0) {
        float *mine = s.row_floats(1 + pl.group);
#pragma unroll
        for (int i = 0; i < P::HALVES * P::PAIRS; ++i) mine[pl.row0 + 8 * i] = m[i];
    }
    epilogue_sync();
    const float *all = s.row_floats(1) + pl.row0;
#pragma unroll
    for (int i = 0; i < P::HALVES * P::PAIRS; ++i)
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
        for (int i = 0; i < 16; ++i)
            if (((i >> 1) & 1) < P::PAIRS) m[2 * half + ((i >> 1) & 1)] = fmaxf(m[2 * half + ((i >> 1) & 1)], fabsf(x[half][i]));
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
        const float2 b = P::PAIRS == 2 && r1 < N ? *reinterpret_cast<const float2 *>(p1 + 8 * j) : make_float2(0.f, 0.f);
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
        if (P::PAIRS == 2 && r1 < N) *reinterpret_cast<float2 *>(p1 + 8 * j) = make_float2(v[4 * j + 2], v[4 * j + 3]);
    }
}

// Loads a tile of rows as an operand: warp w takes rows EACH w .., lane l the columns 4 l .. 4 l + 3 (fetch(row,
// lane) returns them); the row's scale comes from its own largest magnitude, 1 / scale goes to row_floats(0).
template <class P, class Fetch>
__device__ __forceinline__ void load_operand(const Shared &s, unsigned char *buf, Fetch &&fetch)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *inv_out = s.row_floats(0);
    constexpr int EACH = P::EACH;
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
// Rows of a tile: as few as leave an SM for each tile, except where the caller asked for the least SM time (dense_tile_rows 32:
// batches on several streams).  Every epilogue of the chain shortens with the rows; the products, which are not what it waits for,
// take as long as before.  Median of a network's boundaries (inference; training forward; backward): 391 rows in tiles of 32 and 64
// 18 and 21, 20 and 24, 21 and 28 us; 2,701 rows 20 and 22, 22 and 26, 22 and 29; 4,881 rows in tiles of 64 and 128 24 and 31, 30 and
// 39, 33 and 48; 9,301 rows 32 and 32, 34 and 49, 35 and 52.  (A cluster of four blocks on a tile of 128 rows, each with a hidden
// chunk and one of q, k, v: 21, 22 and 29 us at 391 rows; what it saved of the products went into the exchange.)
// More tiles than SMs follow one another: two of 64 rows take longer than one of 128.
inline int tile_rows(long long rows)
{
    const long long sms = sm_count();
    return dense_tile_rows_choice() == 32 || rows > 64 * sms ? 128 : rows > 32 * sms ? 64 : 32;
}

// Shared memory of a launch's kernels, once per thread and device.
struct DenseLaunch {
    bool configured[64] = {};
    int configure(const void *const (&kernels)[3], const char *what)
    {
        int dev = 0;
        cudaGetDevice(&dev);
        if (configured[dev & 63]) return CF_OK;
        for (const void *kernel : kernels)
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) {
                cudaGetLastError();
                return fail(CF_ERR_CUDA, "%s: %d bytes of shared memory not available", what, SMEM_BYTES);
            }
        configured[dev & 63] = true;
        return CF_OK;
    }
};

}  // namespace tc5
}  // namespace cf
