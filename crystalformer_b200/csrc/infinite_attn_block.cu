// Fused infinitely connected attention, forward, eight query rows of a crystal per thread block.
//
// The row kernel (infinite_attn_fwd.cu) reads every key's k and v for every query: 1 KB per edge, which at crystals of
// 100-200 atoms is 1.5 GB of L2 traffic per call and most of its time; at small crystals its four warps per row spend
// their time in the barriers between the row's phases.  Here a block holds eight rows of one crystal, so k and v are read
// once per eight rows, and the long phase - the sweep over a row's (key, translation) terms - is one warp per row with
// no barrier in it; two blocks per SM fill each other's barriers (sixteen rows in one block had nothing beside them).  Phases:
//   1  s_h[j] = q_i.k_j for all rows, keys and heads into shared memory           (warp = head, lane = key)
//   2  phi from the edge's term list (term_list.cuh), logit = s + phi to global memory, soft-max statistics
//                                                                                 (thread = row and key)
//   3  Psi_i over the row's listed terms with the joint weight exp(s - lse + a d2) (warp = row; lanes = terms, then bins)
//   4  p = exp(logit - lse) over s in shared memory, sum_j p v_j + W Psi          (warp = head)
// Rows without a term list are left to the row kernel (their phi is written all the same).  Every sum has a fixed order.
#include "infinite_attn_block.cuh"
#include "lattice_core.cuh"
#include "term_list.cuh"

namespace cf {
int launch_listless_rows(const float *q, const float *k, const float *v, const float *a, const float *pos_ij, const float *tvecs,
                         const float *rvlen, const int64_t *batch, const int64_t *edges, const int64_t *row_start, int64_t N, int64_t E,
                         int64_t max_atoms, double dist_max, double wscale, const float *W, double cutoff_radius, int lattice_range,
                         int minimum_range, float *out, float *logit, float *lse, float *psi_row, const TermList &list, const int *rows,
                         const unsigned *count, unsigned *ticket, int64_t K, cudaStream_t s);
namespace {

constexpr int BR_ROWS = 8;
constexpr int BR_THREADS = 256;
constexpr int BR_WARPS = 8;
constexpr int BR_LD = 12;      // floats per (head, key) of the s / p table: 8 rows, 16-byte aligned, spread over the banks
constexpr int BR_RING = 64;    // candidates: up to 31 left over + 32 offered
constexpr int BR_WARP_FLOATS = STAGE_FLOATS + 2 * BR_RING;
constexpr int PSI_LD = 68;     // floats per (row, head) of the Psi tile
constexpr int CH = HEADS * HEAD_DIM;

struct BlockArgs {
    const float *q, *k, *v, *a, *pos_ij, *tvecs, *rvlen, *W;
    const int64_t *batch, *edges, *row_start;
    const int *blocks;            // first atom of every block of rows
    const unsigned *block_count;
    unsigned *ticket;             // zero on entry
    int *leftover;                // rows without a list
    unsigned *leftover_count;     // zero on entry
    TermList list;
    long long E;
    float *out, *logit, *lse, *psi_row;
    int max_atoms;
    BoxRule rule;
    BasisParams basis;
};

__host__ __device__ constexpr int key_stride(int max_atoms) { return (max_atoms + 1) & ~1; }
template <bool PSI>
__host__ __device__ constexpr size_t block_floats(int max_atoms)
{
    // s / p table; Psi tile (before it: the partial soft-max statistics, 32 x 8 x 8 x 2); per warp the staging area and the
    // candidate ring (before them: the queries); per (row, head): a log2e, box, -lse log2e
    return (size_t)HEADS * key_stride(max_atoms) * BR_LD + (PSI ? BR_ROWS * HEADS * PSI_LD : 2 * 32 * BR_ROWS * HEADS) +
           (PSI ? BR_WARPS * BR_WARP_FLOATS : BR_ROWS * CH) + 3 * BR_ROWS * HEADS;
}
// two blocks per SM (228 KB, of which a block takes 1 KB for itself) up to ROW_BLOCK_MAX_ATOMS, and no further
constexpr size_t two_blocks(int max_atoms) { return 2 * (sizeof(float) * block_floats<true>(max_atoms) + 16 + 1024); }
static_assert(two_blocks(ROW_BLOCK_MAX_ATOMS) <= 233472 && two_blocks(ROW_BLOCK_MAX_ATOMS + 1) > 233472, "the largest crystal of two blocks per SM");
static_assert(BR_ROWS * CH <= BR_WARPS * BR_WARP_FLOATS, "the queries fit where the warps' buffers will be");
static_assert(2 * 32 * BR_ROWS * HEADS <= BR_ROWS * HEADS * PSI_LD, "the statistics fit where the Psi tile will be");

// phi of one edge by enumeration (no list, or a head whose box misses every listed term): out of line
__device__ __noinline__ void block_phi_enumerated(const BoxRule rule, const float *a_row, const float *rvlen3, const float *tvecs9,
                                                  const float *pos3, float floor_log2, float *z_out)
{
    float a[8], z[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) a[h] = a_row[h];
    Cell cell;
    cell.load(tvecs9);
    edge_phi<1>(rule, a, rvlen3, cell, pos3[0], pos3[1], pos3[2], floor_log2, 0, z);
#pragma unroll
    for (int h = 0; h < 8; ++h) z_out[h] = z[h];
}

template <bool PSI>
__global__ void __launch_bounds__(BR_THREADS, 2) infinite_attn_block_kernel(const BlockArgs p)
{
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kst = key_stride(p.max_atoms);
    float *s = smem;                                            // [8][kst][BR_LD]
    float *psi = s + (size_t)HEADS * kst * BR_LD;               // [8][8][PSI_LD]
    float *stats = psi;                                         // [32][8][8][2], before the tile is filled
    float *stage_all = psi + (PSI ? BR_ROWS * HEADS * PSI_LD : 2 * 32 * BR_ROWS * HEADS);
    float *qs = stage_all;                                      // [8][128], before the warps' buffers are used
    float *a2s = stage_all + (PSI ? BR_WARPS * BR_WARP_FLOATS : BR_ROWS * CH);  // [8][8] a log2e
    int *boxes = reinterpret_cast<int *>(a2s + BR_ROWS * HEADS);  // [8][8]
    float *nlse = a2s + 2 * BR_ROWS * HEADS;                    // [8][8] -lse log2e
    __shared__ unsigned next_sh;
    BinAccumulator<64> bins;
    CandidateRingOf<BR_RING> ring;
    if (PSI) {
        bins.init(stage_all + warp * BR_WARP_FLOATS, lane, p.basis);
        ring.init(stage_all + warp * BR_WARP_FLOATS + STAGE_FLOATS, lane);
    }
    grid_launch_dependents();
    grid_dependency_wait();
    const unsigned count = *p.block_count;
    unsigned at = blockIdx.x;
    while (at < count) {
        if (tid == 0) next_sh = gridDim.x + atomicAdd(p.ticket, 1u);
        const long long i0 = p.blocks[at];
        const long long c = p.batch[i0], e00 = p.row_start[i0];
        const int n = (int)(p.row_start[i0 + 1] - e00);
        const long long a0 = p.edges[p.E + e00];
        const int rows = (int)min((long long)BR_ROWS, a0 + n - i0);
        const float *rvlen3 = p.rvlen ? p.rvlen + 3 * c : nullptr;
        const float *kmat = p.k + a0 * CH;
        // ---- queries, widths and boxes of the rows
        for (int idx = tid; idx < rows * 32; idx += BR_THREADS)
            reinterpret_cast<float4 *>(qs)[idx] = __ldg(reinterpret_cast<const float4 *>(p.q + i0 * CH) + idx);
        if (tid < rows * HEADS) {
            const float a = p.a[i0 * HEADS + tid];
            a2s[tid] = a * LOG2E;
            boxes[tid] = packed_box(p.rule, a, rvlen3);
        }
        __syncthreads();
        // ---- 1: s
        for (int j0 = 0; j0 < n; j0 += 32) {
            const int h = warp, j = j0 + lane;
            const float4 *kp = reinterpret_cast<const float4 *>(kmat + (size_t)min(j, n - 1) * CH + h * HEAD_DIM);
            const float4 k0 = __ldg(kp), k1 = __ldg(kp + 1), k2 = __ldg(kp + 2), k3 = __ldg(kp + 3);
            float *dst = s + ((size_t)h * kst + j) * BR_LD;
#pragma unroll
            for (int r0 = 0; r0 < BR_ROWS; r0 += 4) {
                if (r0 >= rows) break;
                float d[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 *qp = reinterpret_cast<const float4 *>(qs + (r0 + u) * CH + h * HEAD_DIM);
                    const float4 q0 = qp[0], q1 = qp[1], q2 = qp[2], q3 = qp[3];
                    float t0 = q0.x * k0.x, t1 = q2.x * k2.x;
                    t0 = fmaf(q0.y, k0.y, t0); t0 = fmaf(q0.z, k0.z, t0); t0 = fmaf(q0.w, k0.w, t0);
                    t0 = fmaf(q1.x, k1.x, t0); t0 = fmaf(q1.y, k1.y, t0); t0 = fmaf(q1.z, k1.z, t0); t0 = fmaf(q1.w, k1.w, t0);
                    t1 = fmaf(q2.y, k2.y, t1); t1 = fmaf(q2.z, k2.z, t1); t1 = fmaf(q2.w, k2.w, t1);
                    t1 = fmaf(q3.x, k3.x, t1); t1 = fmaf(q3.y, k3.y, t1); t1 = fmaf(q3.z, k3.z, t1); t1 = fmaf(q3.w, k3.w, t1);
                    d[u] = t0 + t1;
                }
                if (j < n) *reinterpret_cast<float4 *>(dst + r0) = make_float4(d[0], d[1], d[2], d[3]);
            }
        }
        __syncthreads();
        // ---- 2: phi and the soft-max statistics; thread = (row r, key group jg)
        const int r = tid & 7, jg = tid >> 3;
        {
            float M[8], L[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) { M[h] = -INFINITY; L[h] = 0.f; }
            if (r < rows) {
                float a2[8];
                int pk[8];
                float a2max = -INFINITY;
#pragma unroll
                for (int h = 0; h < 8; ++h) {
                    a2[h] = a2s[r * HEADS + h];
                    pk[h] = boxes[r * HEADS + h];
                    a2max = fmaxf(a2max, a2[h]);
                }
                const bool listed = p.list.start[e00 + (long long)r * n] >= 0;
                for (int j = jg; j < n; j += 32) {
                    const long long e = e00 + (long long)r * n + j;
                    const int first = p.list.start[e];
                    const int cnt = first >= 0 ? p.list.count[e] : 0;
                    const float m = first >= 0 ? p.list.dmin[e] : 0.f;
                    const float2 *ent = p.list.pool + (first >= 0 ? first : 0);
                    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    float2 n0 = make_float2(0.f, 0.f), n1 = n0;  // entries are requested two steps ahead of their use
                    if (0 < cnt) n0 = __ldg(ent);
                    if (1 < cnt) n1 = __ldg(ent + 1);
                    for (int t = 0; t < cnt; ++t) {
                        const float2 en = n0;
                        n0 = n1;
                        if (t + 2 < cnt) n1 = __ldg(ent + t + 2);
                        const float rel = en.x - m;
                        if (a2max * rel < p.basis.floor_log2) continue;  // below the floor for every head
                        const int key = __float_as_int(en.y);
#pragma unroll
                        for (int h = 0; h < 8; ++h)
                            if (key_in_box(key, pk[h])) sum[h] += ex2(a2[h] * rel);
                    }
                    float phi[8];
                    bool done = cnt > 0;
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        phi[h] = fmaf(m, a2[h] * LN2, logf(sum[h]));
                        done = done && sum[h] > 1e-30f;
                    }
                    if (!done) block_phi_enumerated(p.rule, p.a + (i0 + r) * HEADS, rvlen3, p.tvecs + 9 * c, p.pos_ij + 3 * e, p.basis.floor_log2, phi);
                    float lg[8];
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        lg[h] = s[((size_t)h * kst + j) * BR_LD + r] + phi[h];
                        const float x = lg[h] * LOG2E, top = fmaxf(M[h], x);
                        L[h] = fmaf(L[h], ex2(M[h] - top), ex2(x - top));
                        M[h] = top;
                    }
                    float4 *dst = reinterpret_cast<float4 *>(p.logit + e * HEADS);  // (phi alone for the row kernel, if the row goes there)
                    dst[0] = listed ? make_float4(lg[0], lg[1], lg[2], lg[3]) : make_float4(phi[0], phi[1], phi[2], phi[3]);
                    dst[1] = listed ? make_float4(lg[4], lg[5], lg[6], lg[7]) : make_float4(phi[4], phi[5], phi[6], phi[7]);
                }
            }
            float4 *st = reinterpret_cast<float4 *>(stats + ((size_t)jg * BR_ROWS + r) * 16);
#pragma unroll
            for (int t = 0; t < 4; ++t) st[t] = make_float4(M[2 * t], L[2 * t], M[2 * t + 1], L[2 * t + 1]);
        }
        __syncthreads();
        if (tid < rows * HEADS) {  // (r, h): the 32 groups' statistics in their order
            const float2 *st = reinterpret_cast<const float2 *>(stats) + tid;
            float M = -INFINITY, L = 0.f;
#pragma unroll 8
            for (int g = 0; g < 32; ++g) M = fmaxf(M, st[(size_t)g * BR_ROWS * HEADS].x);
#pragma unroll 8
            for (int g = 0; g < 32; ++g) {
                const float2 v = st[(size_t)g * BR_ROWS * HEADS];
                L = fmaf(v.y, ex2(v.x - M), L);
            }
            const float l2 = M + log2f(L);
            nlse[tid] = -l2;
            p.lse[i0 * HEADS + tid] = l2 * LN2;
        }
        __syncthreads();
        // ---- 3: the row's terms
        if (PSI && warp < rows) {
            const long long e0 = e00 + (long long)warp * n;
            const int list_first = p.list.start[e0];
            if (list_first < 0) {
                if (lane == 0) p.leftover[atomicAdd(p.leftover_count, 1u)] = (int)(i0 + warp);
            } else {
                float a2[8], nl[8];
                int pk[8];
                float a2max = -INFINITY;
                int uni = 0;
#pragma unroll
                for (int h = 0; h < 8; ++h) {
                    a2[h] = a2s[warp * HEADS + h];
                    nl[h] = nlse[warp * HEADS + h];
                    pk[h] = boxes[warp * HEADS + h];
                    a2max = fmaxf(a2max, a2[h]);
                    uni = box_union(uni, pk[h]);
                }
                bool masked = false;
#pragma unroll
                for (int h = 0; h < 8; ++h) masked = masked || pk[h] != uni;
                // an upper bound of every term's offset: the largest s - lse of the row
                const float *srow = s + warp;
                float cmax = -INFINITY;
                for (int j = lane; j < n; j += 32)
#pragma unroll
                    for (int h = 0; h < 8; ++h) cmax = fmaxf(cmax, fmaf(srow[((size_t)h * kst + j) * BR_LD], LOG2E, nl[h]));
                cmax = warp_max(cmax);
                bins.clear();
                auto consume = [&]() {
                    float d2;
                    int key;
                    const bool got = ring.take(d2, key);
                    const int j = got ? (key & 2047) : 0;
                    float w[8];
                    float emax = -INFINITY;
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        float eh = fmaf(a2[h], d2, fmaf(srow[((size_t)h * kst + j) * BR_LD], LOG2E, nl[h]));
                        if (!got || (masked && !key_in_box(key, pk[h]))) eh = -INFINITY;
                        w[h] = ex2(eh);
                        emax = fmaxf(emax, eh);
                    }
                    bins.push(emax > p.basis.floor_log2, fast_sqrt(d2) * p.basis.bin_scale, w);
                };
                const int list_end = p.list.start[e0 + n - 1] + p.list.count[e0 + n - 1];
                float2 ahead = make_float2(0.f, 0.f);
                if (list_first + lane < list_end) ahead = __ldg(p.list.pool + list_first + lane);
                for (int first = list_first; first < list_end; first += 32) {
                    const bool live = first + lane < list_end;
                    const float2 en = ahead;
                    if (first + 32 + lane < list_end) ahead = __ldg(p.list.pool + first + 32 + lane);
                    const int key = __float_as_int(en.y);
                    // (the lists are built for a box that contains every head's: terms outside this row's boxes drop out here)
                    ring.offer(live && key_in_box(key, uni) && fmaf(a2max, en.x, cmax) > p.basis.floor_log2 && en.x < p.basis.d2_cut,
                               en.x, key);
                    while (ring.ready()) consume();
                }
                while (ring.count > 0) consume();
                float *mine = psi + (size_t)warp * HEADS * PSI_LD;
                bins.flush(mine, PSI_LD);
                if (p.psi_row) {
                    float4 *dst = reinterpret_cast<float4 *>(p.psi_row + (i0 + warp) * HEADS * 64) + lane;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        dst[32 * t] = *reinterpret_cast<const float4 *>(mine + (2 * t + (lane >> 4)) * PSI_LD + 4 * (lane & 15));
                }
            }
        }
        if (!PSI && tid < rows && p.list.start[e00 + (long long)tid * n] < 0)
            p.leftover[atomicAdd(p.leftover_count, 1u)] = (int)(i0 + tid);
        __syncthreads();
        // ---- 4: p over s, then the weighted sums
        if (r < rows) {
            for (int j = jg; j < n; j += 32) {
                const float4 *src = reinterpret_cast<const float4 *>(p.logit + (e00 + (long long)r * n + j) * HEADS);
                const float4 x = src[0], y = src[1];
                const float lg[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                for (int h = 0; h < 8; ++h) s[((size_t)h * kst + j) * BR_LD + r] = ex2(fmaf(lg[h], LOG2E, nlse[r * HEADS + h]));
            }
        }
        __syncthreads();
        {
            const int h = warp, d = lane & 15, par = lane >> 4;
            {
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                const float *vp = p.v + a0 * CH + h * HEAD_DIM + d;
                const float *pp = s + (size_t)h * kst * BR_LD;
#pragma unroll 4
                for (int j = par; j < n; j += 2) {
                    const float v = __ldg(vp + (size_t)j * CH);
                    const float4 x = *reinterpret_cast<const float4 *>(pp + (size_t)j * BR_LD), y = *reinterpret_cast<const float4 *>(pp + (size_t)j * BR_LD + 4);
                    acc[0] = fmaf(x.x, v, acc[0]); acc[1] = fmaf(x.y, v, acc[1]); acc[2] = fmaf(x.z, v, acc[2]); acc[3] = fmaf(x.w, v, acc[3]);
                    acc[4] = fmaf(y.x, v, acc[4]); acc[5] = fmaf(y.y, v, acc[5]); acc[6] = fmaf(y.z, v, acc[6]); acc[7] = fmaf(y.w, v, acc[7]);
                }
                if (PSI) {
                    const float4 *w4 = reinterpret_cast<const float4 *>(p.W + (size_t)(h * HEAD_DIM + d) * 64 + 32 * par);
                    const float *ps = psi + (size_t)h * PSI_LD + 32 * par;
#pragma unroll 2
                    for (int k4 = 0; k4 < 8; ++k4) {
                        const float4 w = __ldg(w4 + k4);
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const float4 x = *reinterpret_cast<const float4 *>(ps + (size_t)u * HEADS * PSI_LD + 4 * k4);
                            acc[u] = fmaf(w.x, x.x, acc[u]); acc[u] = fmaf(w.y, x.y, acc[u]);
                            acc[u] = fmaf(w.z, x.z, acc[u]); acc[u] = fmaf(w.w, x.w, acc[u]);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    acc[u] += __shfl_xor_sync(FULL, acc[u], 16);
                    if ((u >> 2) == par && u < rows) p.out[(i0 + u) * CH + h * HEAD_DIM + d] = acc[u];
                }
            }
        }
        __syncthreads();
        at = next_sh;
        __syncthreads();  // (the next block's ticket is drawn after everybody has read this one)
    }
}

// The blocks of rows: the atoms whose place in their crystal is a multiple of eight, about in the order of row_order.
__global__ void row_blocks_kernel(const int32_t *row_order, const int64_t *row_start, const int64_t *edges, long long E, long long N,
                                  int *blocks, unsigned *count)
{
    const long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= N) return;
    const long long i = row_order ? row_order[at] : at;
    const long long e0 = row_start[i];
    if (row_start[i + 1] > e0 && (i - edges[E + e0]) % BR_ROWS == 0) blocks[atomicAdd(count, 1u)] = (int)i;
}

}  // namespace

int launch_row_blocks(const RowBlocks &b, const int32_t *row_order, const int64_t *row_start, const int64_t *edges, long long N, long long E,
                      cudaStream_t s)
{
    if (cudaMemsetAsync(b.counters, 0, sizeof(unsigned) * 4 * (ROW_BLOCK_LAYERS + 1), s) != cudaSuccess) return launch_status("row blocks");
    row_blocks_kernel<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(row_order, row_start, edges, E, N, b.blocks, b.counters);
    return launch_status("row_blocks_kernel");
}

int block_attn_impl(const float *q, const float *k, const float *v, const float *a, const float *pos_ij, const float *tvecs,
                    const float *rvlen, const int64_t *batch, const int64_t *edges, const int64_t *row_start, int64_t N, int64_t B,
                    int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale, const float *W, double cutoff_radius,
                    int lattice_range, int minimum_range, float *out, float *logit, float *lse, float *psi_row, const TermList &list,
                    const RowBlocks &blocks, int call, cudaStream_t s)
{
    CF_REQUIRE(max_atoms >= 1 && max_atoms <= ROW_BLOCK_MAX_ATOMS && call >= 0 && call < ROW_BLOCK_LAYERS && list.pool != nullptr, CF_ERR_INVALID,
               "row block attention: max_atoms=%lld (1..%d), call %d", (long long)max_atoms, ROW_BLOCK_MAX_ATOMS, call);
    unsigned *counters = blocks.counters + 4 * (call + 1);
    BlockArgs p{};
    p.q = q; p.k = k; p.v = v; p.a = a; p.pos_ij = pos_ij; p.tvecs = tvecs; p.rvlen = cutoff_radius != 0.0 ? rvlen : nullptr; p.W = W;
    p.batch = batch; p.edges = edges; p.row_start = row_start;
    p.blocks = blocks.blocks; p.block_count = blocks.counters; p.ticket = counters; p.leftover = blocks.leftover; p.leftover_count = counters + 1;
    p.list = list; p.E = E; p.out = out; p.logit = logit; p.lse = lse; p.psi_row = psi_row; p.max_atoms = (int)max_atoms;
    p.rule = BoxRule{(float)cutoff_radius, lattice_range, minimum_range};
    p.basis = make_basis_params(K, dist_max, wscale, weight_floor_log2());
    const bool with_psi = K > 0;
    const size_t smem = sizeof(float) * (with_psi ? block_floats<true>((int)max_atoms) : block_floats<false>((int)max_atoms));
    auto kernel = with_psi ? infinite_attn_block_kernel<true> : infinite_attn_block_kernel<false>;
    static thread_local size_t configured[64][2] = {};
    static thread_local int occupancy[64][2] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const int slot = with_psi ? 1 : 0;
    if (configured[dev & 63][slot] != smem) {
        int occ = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, BR_THREADS, smem) != cudaSuccess || occ <= 0) {
            cudaGetLastError();
            return fail(CF_ERR_CUDA, "row block attention: %zu bytes of shared memory not available", smem);
        }
        configured[dev & 63][slot] = smem;
        occupancy[dev & 63][slot] = occ;
    }
    // (at most N / 8 + B blocks of rows exist; how many is known on the device)
    const long long most = N / BR_ROWS + B, cap = (long long)sm_count() * occupancy[dev & 63][slot];
    launch_chained(kernel, dim3((unsigned)(most < cap ? (most > 0 ? most : 1) : cap)), dim3(BR_THREADS), smem, s, true, p);
    int rc = launch_status("infinite_attn_block_kernel");
    if (rc == CF_OK)
        rc = launch_listless_rows(q, k, v, a, pos_ij, tvecs, p.rvlen, batch, edges, row_start, N, E, max_atoms, dist_max, wscale, W, cutoff_radius,
                                  lattice_range, minimum_range, out, logit, lse, psi_row, list, blocks.leftover, counters + 1, counters + 2, K, s);
    return rc;
}

}  // namespace cf
