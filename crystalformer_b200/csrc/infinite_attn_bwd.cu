// Fused infinitely connected attention, backward.  phi and psi are recomputed from the geometry.
//
// With the joint weight of a (key, translation) term  P_jn = p_ij p(n|ij) = exp(q_i.k_j - lse_i + a_i d2_jn),
// u_i = W^T gout_i (8 x 64), c(d) = sum_k u_i[k] g_k(d), delta_i = gout_i . out_i and gov_j = gout_i . v_j:
//     glogit_ij = p_ij (gov_j - delta_i) + sum_n P_jn c(d_jn)
//     ga_i      = sum_{j,n} P_jn d2_jn (gov_j - delta_i + c(d_jn))          (the products of per-edge sums cancel)
//     gq_i      = sum_j glogit_ij k_j          gk_j = sum_i glogit_ij q_i          gv_j = sum_i p_ij gout_i
// which is the chain of models/kernels/fused_dpa_bwd.cu:53-114 and real_enc_proj_bwd.cu:153-218 written for the
// hoisted projection.  The gradient of W is sum_i gout_i (x) psi_row_i, a GEMM done by the caller.
//
//   infinite_attn_bwd_rows_kernel  CTA per atom i: recompute q.k, p_ij, then each warp takes a contiguous range of the
//                                  row's keys.  Lanes run over (key, translation) terms; those within reach of the widest
//                                  head are collected, and every lane takes one: its eight joint weights, the contraction
//                                  of the basis with u_i, and a segmented scan for the sums per key (fixed order, one warp
//                                  per key).  Writes glogit (E,H), ga (N,H), gq (N,H,D).
//   infinite_attn_bwd_cols_kernel  gk_j, gv_j from glogit and p_ij = exp(logit - lse_i), eight keys per block.
#include "lattice_bwd_core.cuh"
#include "pair_grid.cuh"
#include "term_list.cuh"

namespace cf {
namespace {

constexpr int THREADS = 128;
constexpr int WARPS = THREADS / 32;
constexpr int KBINS = 64;
constexpr int BWD_RING = 64;  // candidates of a warp: up to 31 left over + 32 offered

struct BwdRowArgs {
    const float *q, *k, *v, *a, *pos, *pos_ij, *tvecs, *rvlen, *W, *logit, *lse, *out, *gout;
    const int64_t *batch, *edges, *row_start;
    const int32_t *row_order;
    float *gq, *gk, *gv, *ga, *glogit;
    long long N, E;
    int max_atoms;
    BoxRule rule;
    BasisParams basis;
    TermList list;  // optional (pool == NULL: none): the rows' terms, found once per batch (term_list.cuh)
    const unsigned *rows_on_device;  // optional: the number of rows to process (entries of row_order), read on the device
    bool pieces;    // logit, lse, glogit and prob start on 16 bytes (a caller's may lie anywhere)
    float *prob;    // optional (E,H): p_ij, written by the rows and read by the columns instead of exp(logit - lse)
};

__host__ __device__ inline size_t bwd_row_smem_floats(int max_atoms, bool with_basis)
{
    // per atom: rel (4) + c (8) + p (8) + gov (8) + s0 (8); then u (8 x 64), per-warp candidates, ga partials
    return (size_t)max_atoms * 36 + (with_basis ? HEADS * U_STRIDE : 0) + WARPS * 2 * BWD_RING + WARPS * 8;
}

template <int K, bool LEFT>
__global__ void __launch_bounds__(THREADS, 4) infinite_attn_bwd_rows_kernel(const BwdRowArgs p)
{
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4 *rel = reinterpret_cast<float4 *>(smem);                    // [max_atoms]
    float *cj = smem + (size_t)p.max_atoms * 4;                        // [max_atoms][8] (q.k - lse) log2e
    float *pj = cj + (size_t)p.max_atoms * 8;                          // [max_atoms][8] p_ij
    float *gov = pj + (size_t)p.max_atoms * 8;                         // [max_atoms][8] gout_i . v_j - delta_i
    float *s0 = gov + (size_t)p.max_atoms * 8;                         // [max_atoms][8] sum_n P c, then glogit
    float *u = s0 + (size_t)p.max_atoms * 8;                           // [8][64]
    float *rings = u + (K > 0 ? HEADS * U_STRIDE : 0);                 // [WARPS][2 BWD_RING]
    float *ga_part = rings + WARPS * 2 * BWD_RING;                     // [WARPS][8]
    CandidateRingOf<BWD_RING> ring;
    ring.init(rings + warp * 2 * BWD_RING, lane);

    const long long rows = LEFT ? (long long)*p.rows_on_device : p.N;
    // what a row starts from: atom, edges, keys, first key; fetched a row ahead (dependent reads)
    struct Row {
        long long i, e0, a0;
        int n;
    };
    auto row_of = [&](long long slot) {
        Row r{0, 0, 0, 0};
        if (slot < rows) {
            r.i = p.row_order ? p.row_order[slot] : slot;
            r.e0 = p.row_start[r.i];
            r.n = (int)(p.row_start[r.i + 1] - r.e0);
            r.a0 = r.n > 0 ? p.edges[p.E + r.e0] : 0;
        }
        return r;
    };
    Row next = row_of(blockIdx.x);
    for (long long slot = blockIdx.x; slot < rows; slot += gridDim.x) {
        const long long i = next.i, e0 = next.e0, a0 = next.a0;
        const int n = next.n;
        const long long c = p.batch[i];
        next = row_of(slot + gridDim.x);
        if (n > p.max_atoms) {
            p.gq[i * HEADS * HEAD_DIM + tid] = __int_as_float(0x7fc00000);
            if (tid < HEADS) p.ga[i * HEADS + tid] = __int_as_float(0x7fc00000);
            continue;
        }
        // ---- per key: (q.k - lse) log2e, p_ij, gout_i.v_j - delta_i.  A key's k and v rows are one coalesced read of a warp
        //      each (lane l: channels 4 l .. 4 l + 3, head l / 4); the four lanes of a head add their partial products, and
        //      then take one of the four results each.  delta_i = gout_i . out_i in every warp.  (One key per lane read
        //      each of its 16-byte pieces from a line of its own: 60 % of the L1's wavefronts.)
        {
            const float4 q4 = __ldg(reinterpret_cast<const float4 *>(p.q + i * HEADS * HEAD_DIM) + lane);
            const float4 go = __ldg(reinterpret_cast<const float4 *>(p.gout + i * HEADS * HEAD_DIM) + lane);
            const float4 ou = __ldg(reinterpret_cast<const float4 *>(p.out + i * HEADS * HEAD_DIM) + lane);
            const int h = lane >> 2, t = lane & 3;
            const float lse = p.lse[i * HEADS + h];
            const float4 *kp = reinterpret_cast<const float4 *>(p.k + a0 * HEADS * HEAD_DIM) + lane;
            const float4 *vp = reinterpret_cast<const float4 *>(p.v + a0 * HEADS * HEAD_DIM) + lane;
            float delta = fmaf(go.w, ou.w, fmaf(go.z, ou.z, fmaf(go.y, ou.y, go.x * ou.x)));
            delta += __shfl_xor_sync(FULL, delta, 1);
            delta += __shfl_xor_sync(FULL, delta, 2);
            for (int j0 = 4 * warp; j0 < n; j0 += 4 * WARPS) {
                float4 kk[4], vv[4];
                float lg[4];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const int j = min(j0 + w, n - 1);
                    kk[w] = __ldg(kp + (size_t)j * 32);
                    vv[w] = __ldg(vp + (size_t)j * 32);
                    lg[w] = t == 2 ? p.logit[(e0 + j) * HEADS + h] : 0.f;
                }
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    float s = fmaf(q4.w, kk[w].w, fmaf(q4.z, kk[w].z, fmaf(q4.y, kk[w].y, q4.x * kk[w].x)));
                    float g = fmaf(go.w, vv[w].w, fmaf(go.z, vv[w].z, fmaf(go.y, vv[w].y, go.x * vv[w].x)));
                    s += __shfl_xor_sync(FULL, s, 1);
                    g += __shfl_xor_sync(FULL, g, 1);
                    s += __shfl_xor_sync(FULL, s, 2);
                    g += __shfl_xor_sync(FULL, g, 2);
                    const float x = ((t == 0 ? s : lg[w]) - lse) * LOG2E;
                    const float val = t == 0 ? x : t == 1 ? g - delta : t == 2 ? ex2(x) : 0.f;
                    float *dst = (t == 0 ? cj : t == 1 ? gov : t == 2 ? pj : s0) + (j0 + w) * 8 + h;
                    if (j0 + w < n) *dst = val;
                }
            }
        }
        // ---- relative positions (rows without a list), u_i = W^T gout_i: thread = head and four bins
        const int list_first = (p.list.pool != nullptr && n > 0) ? p.list.start[e0] : -1;
        if (list_first < 0) {
            const float pix = p.pos_ij ? 0.f : p.pos[3 * i], piy = p.pos_ij ? 0.f : p.pos[3 * i + 1], piz = p.pos_ij ? 0.f : p.pos[3 * i + 2];
            for (int j = tid; j < n; j += THREADS) {
                const float *pp = p.pos_ij ? p.pos_ij + 3 * (e0 + j) : p.pos + 3 * (a0 + j);
                rel[j] = p.pos_ij ? make_float4(pp[0], pp[1], pp[2], 0.f)
                                  : make_float4(__fsub_rn(pp[0], pix), __fsub_rn(pp[1], piy), __fsub_rn(pp[2], piz), 0.f);
            }
        }
        if (K > 0) {
            const int h = tid >> 4, k4 = tid & 15;
            const float4 *go4 = reinterpret_cast<const float4 *>(p.gout + (i * HEADS + h) * HEAD_DIM);
            const float4 *w4 = reinterpret_cast<const float4 *>(p.W + (size_t)h * HEAD_DIM * KBINS) + k4;
            float2 lo = make_float2(0.f, 0.f), hi = lo;
#pragma unroll
            for (int m4 = 0; m4 < HEAD_DIM / 4; ++m4) {
                const float4 g4 = __ldg(go4 + m4);
                const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const float4 w = __ldg(w4 + (4 * m4 + m) * (KBINS / 4));
                    lo = fma2(make_float2(w.x, w.y), make_float2(g[m], g[m]), lo);
                    hi = fma2(make_float2(w.z, w.w), make_float2(g[m], g[m]), hi);
                }
            }
            *reinterpret_cast<float4 *>(u + h * U_STRIDE + 4 * k4) = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
        __syncthreads();

        // ---- main pass: each warp takes a contiguous range of keys and all their translations
        const float a_own = p.a[i * HEADS + (lane & 7)];
        const int pk_own = packed_box(p.rule, a_own, p.rvlen ? p.rvlen + 3 * c : nullptr);
        int uni = pk_own;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) uni = box_union(uni, __shfl_xor_sync(FULL, uni, o));
        const bool masked = !__all_sync(FULL, pk_own == uni);
        float a2[8];
        int pk[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            a2[h] = __shfl_sync(FULL, a_own, h) * LOG2E;
            pk[h] = __shfl_sync(FULL, pk_own, h);
        }
        float a2max = a2[0], cmax = -INFINITY;
#pragma unroll
        for (int h = 1; h < 8; ++h) a2max = fmaxf(a2max, a2[h]);
        for (int idx = lane; idx < n * HEADS; idx += 32) cmax = fmaxf(cmax, cj[idx]);
        cmax = warp_max(cmax);
        float G[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) G[h] = 0.f;
        // one term per lane, terms of a key contiguous: the eight joint weights, their part of ga, and (K > 0) the contraction
        // of the basis with u, summed per key by a segmented scan (a fixed tree over the batch; the last lane of a key's run
        // adds it to the key's total, which no other warp touches)
        auto weigh = [&](bool got, int j, float d2, int key) {
            const float4 ca = *reinterpret_cast<const float4 *>(cj + j * 8);
            const float4 cb = *reinterpret_cast<const float4 *>(cj + j * 8 + 4);
            const float4 ga4 = *reinterpret_cast<const float4 *>(gov + j * 8);
            const float4 gb4 = *reinterpret_cast<const float4 *>(gov + j * 8 + 4);
            const float off[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
            const float gj[8] = {ga4.x, ga4.y, ga4.z, ga4.w, gb4.x, gb4.y, gb4.z, gb4.w};
            float w[8];
            float emax = -INFINITY;
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                float eh = fmaf(a2[h], d2, off[h]);
                if (!got || (masked && !key_in_box(key, pk[h]))) eh = -INFINITY;
                w[h] = ex2(eh);
                emax = fmaxf(emax, eh);
                G[h] = fmaf(w[h] * d2, gj[h], G[h]);
            }
            if (K > 0) {
                const bool keep = emax > p.basis.floor_log2 && d2 < p.basis.d2_cut;
                if (!__any_sync(FULL, keep)) return;
                const float x = fast_sqrt(d2) * p.basis.bin_scale;
                float pc[8];
                if (keep) {
                    if (K == 64 && p.basis.windowed) basis_dot_window(u, x, p.basis.bin_step, pc);
                    else basis_dot<(K > 0 ? K : 4)>(u, x, p.basis.bin_step, pc);
                }
#pragma unroll
                for (int h = 0; h < 8; ++h) {
                    pc[h] = keep ? w[h] * pc[h] : 0.f;
                    G[h] = fmaf(pc[h], d2, G[h]);
                }
                const int id = got ? j : -1;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const bool same = __shfl_up_sync(FULL, id, o) == id && lane >= o && got;
                    if (!__any_sync(FULL, same)) break;  // (no run of equal keys is longer than o)
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        const float up = __shfl_up_sync(FULL, pc[h], o);
                        pc[h] += same ? up : 0.f;
                    }
                }
                const int id_next = __shfl_down_sync(FULL, id, 1);  // (every lane takes part; lane 31 gets its own)
                if (got && (lane == 31 || id_next != id)) {
                    float4 *dst = reinterpret_cast<float4 *>(s0 + j * 8);
                    const float4 x0 = dst[0], x1 = dst[1];
                    dst[0] = make_float4(x0.x + pc[0], x0.y + pc[1], x0.z + pc[2], x0.w + pc[3]);
                    dst[1] = make_float4(x1.x + pc[4], x1.y + pc[5], x1.z + pc[6], x1.w + pc[7]);
                }
                __syncwarp();
            }
        };
        // candidates: terms that the widest head and the row's largest offset could bring above the floor
        auto consume = [&]() {
            float d2;
            int key;
            const bool got = ring.take(d2, key);
            weigh(got, got ? (key & 2047) : 0, got ? d2 : 0.f, key);  // (a lane without an entry reads whatever the ring held)
        };
        if (list_first >= 0) {
            // ---- terms from the row's list (entries contiguous, keys ascending).  A warp takes whole keys, so that
            //      every per-key sum has one owner: warp w gets the keys whose first entry lies in its equal share
            const int list_end = p.list.start[e0 + n - 1] + p.list.count[e0 + n - 1];
            const int span = list_end - list_first, share = (span + WARPS - 1) / WARPS;
            auto keys_before = [&](int target) {  // number of keys whose entries start before `target` (warp-uniform)
                int cnt = 0;
                for (int j0 = 0; j0 < n; j0 += 32) {
                    const int j = j0 + lane;
                    const bool before = j < n && p.list.start[e0 + j] - list_first < target;
                    cnt += __popc(__ballot_sync(FULL, before));
                }
                return cnt;
            };
            const int k_lo = warp == 0 ? 0 : keys_before(warp * share);
            const int k_hi = warp == WARPS - 1 ? n : keys_before((warp + 1) * share);
            const int w_lo = k_lo < n ? p.list.start[e0 + k_lo] : list_end;
            const int w_hi = k_hi < n ? p.list.start[e0 + k_hi] : list_end;
            float2 ahead = make_float2(0.f, 0.f);  // the entries of the next step, requested one step early
            if (w_lo + lane < w_hi) ahead = __ldg(p.list.pool + w_lo + lane);
            for (int at = w_lo; at < w_hi; at += 32) {
                const bool live = at + lane < w_hi;
                const float2 en = ahead;
                if (at + 32 + lane < w_hi) ahead = __ldg(p.list.pool + at + 32 + lane);
                const int key = __float_as_int(en.y);
                // (the lists are built for a box that contains every head's: terms outside this row's boxes drop out here)
                ring.offer(live && key_in_box(key, uni) && fmaf(a2max, en.x, cmax) > p.basis.floor_log2, en.x, key);
                while (ring.ready()) consume();
            }
        } else {
            const int R1 = box_r1(uni), R2 = box_r2(uni), R3 = box_r3(uni);
            const unsigned per_key = (unsigned)((2 * R1 + 1) * (2 * R2 + 1) * (2 * R3 + 1));
            const int keys_per_warp = (n + WARPS - 1) / WARPS;
            const int j_begin = min(warp * keys_per_warp, n), j_end = min(j_begin + keys_per_warp, n);
            const unsigned begin = (unsigned)j_begin * per_key, end = (unsigned)j_end * per_key;
            Cell cell;
            cell.load(p.tvecs + 9 * c);
            const float F1 = (float)R1, F2 = (float)R2, F3 = (float)R3;
            TermWalker walk;
            walk.init(R1, R2, R3, begin + lane);
            for (unsigned base = begin; base < end; base += 32) {
                const bool valid = base + lane < end;
                const int j = valid ? walk.row : j_begin;
                const float4 r = rel[j];
                const float f1 = walk.u1 - F1, f2 = walk.u2 - F2, f3 = walk.u3 - F3;
                const float dx = fmaf(cell.t3x, f3, fmaf(cell.t2x, f2, fmaf(cell.t1x, f1, r.x)));
                const float dy = fmaf(cell.t3y, f3, fmaf(cell.t2y, f2, fmaf(cell.t1y, f1, r.y)));
                const float dz = fmaf(cell.t3z, f3, fmaf(cell.t2z, f2, fmaf(cell.t1z, f1, r.z)));
                const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                int key = j;
                if (masked) key = pack_key(j, abs(__float2int_rn(f1)), abs(__float2int_rn(f2)), abs(__float2int_rn(f3)));
                ring.offer(valid && fmaf(a2max, d2, cmax) > p.basis.floor_log2, d2, key);
                while (ring.ready()) consume();
                walk.step();
            }
        }
        while (ring.count > 0) consume();
#pragma unroll
        for (int h = 0; h < 8; ++h) G[h] = warp_sum(G[h]);
        if (lane < 8) ga_part[warp * 8 + lane] = pick8(G, lane);
        __syncthreads();
        if (tid < HEADS)
            p.ga[i * HEADS + tid] = (ga_part[tid] + ga_part[8 + tid]) + (ga_part[16 + tid] + ga_part[24 + tid]);
        // ---- glogit_ij = p_ij (gov_j - delta) + S0_ij ; keep it in shared memory for gq
        for (int idx = tid; idx < n * HEADS; idx += THREADS) {
            const float g = fmaf(pj[idx], gov[idx], s0[idx]);
            s0[idx] = g;
            p.glogit[e0 * HEADS + idx] = g;
            if (LEFT) p.prob[e0 * HEADS + idx] = pj[idx];
        }
        __syncthreads();
        {
            const int h = tid >> 4;
            float acc = 0.f;
            const float *kp = p.k + a0 * HEADS * HEAD_DIM + tid;
#pragma unroll 8
            for (int j = 0; j < n; ++j) acc = fmaf(s0[j * 8 + h], __ldg(kp + (size_t)j * HEADS * HEAD_DIM), acc);
            p.gq[i * HEADS * HEAD_DIM + tid] = acc;
        }
        __syncthreads();
    }
}

// gk_j = sum_i glogit_ij q_i, gv_j = sum_i p_ij gout_i with p_ij = exp(logit_ij - lse_i) (PROB: as the rows left it).  Block = eight
// consecutive keys (of one crystal at a time), warp = head: a row's values of the eight keys are contiguous in the n x n block, so
// they are read coalesced, thirty-two rows at a time, and q and gout once for the eight keys (a warp per key and head read them, and
// the columns with a stride, once per key: 0.11 ms against 0.02 ms at crystals of 100-200 atoms).
// Bound by latency (27 MB at 16 crystals of 100-200 atoms, 4 us) and issue: the next rows' values, two 16-byte pieces per thread and
// array, are on their way while these are summed, and q and gout are read sixteen rows at a time at constant offsets.  There 27 us
// (a word per thread and wait, offsets by row: 47; the pieces alone: 37), 256 crystals of up to 40 atoms 16.6 us (18.5).
constexpr int COL_KEYS = 8, COL_ROWS = 32, COL_PIECES = COL_ROWS * COL_KEYS * HEADS / 4 / 256;
constexpr int COL_LD = COL_ROWS * COL_KEYS + 4;  // floats per head (bank skew)
template <bool PROB>
__global__ void __launch_bounds__(256, 3) infinite_attn_bwd_cols_kernel(const BwdRowArgs p)
{
    __shared__ __align__(16) float gs[HEADS * COL_LD], ps[HEADS * COL_LD];
    const int tid = threadIdx.x, lane = tid & 31, h = tid >> 5;
    const int d = lane & 15, par = lane >> 4;
    const int pi = tid >> 4, pj = (tid >> 1) & 7, ph = (tid & 1) * 4;  // the thread's piece: row, key, four heads
    for (long long tile = blockIdx.x; tile * COL_KEYS < p.N; tile += gridDim.x) {
        long long j0 = tile * COL_KEYS;
        const long long tile_end = min(j0 + COL_KEYS, p.N);
        while (j0 < tile_end) {
            const long long r0 = p.row_start[j0];
            const int n = (int)(p.row_start[j0 + 1] - r0);
            if (n == 0) { ++j0; continue; }
            const long long first = p.edges[p.E + r0];
            const long long c0 = p.row_start[first];
            const int jl = (int)(j0 - first), keys = (int)(min(tile_end, first + n) - j0);
            const size_t at = ((size_t)c0 + jl + pj) * HEADS + ph;
            auto four = [&](const float *x) { return p.pieces ? *reinterpret_cast<const float4 *>(x) : make_float4(x[0], x[1], x[2], x[3]); };
            float4 g[COL_PIECES], w[COL_PIECES], ls[COL_PIECES];
            auto fetch = [&](int i0) {
#pragma unroll
                for (int u = 0; u < COL_PIECES; ++u) {
                    const int i = i0 + pi + 16 * u;
                    g[u] = w[u] = ls[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (i < n && pj < keys) {
                        const size_t e = at + (size_t)i * n * HEADS;
                        g[u] = four(p.glogit + e);
                        w[u] = four((PROB ? p.prob : p.logit) + e);
                        if (!PROB) ls[u] = four(p.lse + (first + i) * HEADS + ph);
                    }
                }
            };
            float ak[COL_KEYS], av[COL_KEYS];
#pragma unroll
            for (int u = 0; u < COL_KEYS; ++u) ak[u] = av[u] = 0.f;
            fetch(0);
            for (int i0 = 0; i0 < n; i0 += COL_ROWS) {
                const int rows = min(COL_ROWS, n - i0);
                __syncthreads();  // (the previous chunk has been read)
#pragma unroll
                for (int u = 0; u < COL_PIECES; ++u) {
                    const int o = ph * COL_LD + (pi + 16 * u) * COL_KEYS + pj;
                    const float4 x = w[u];
                    auto prob = [&](float v, float l) { return PROB ? v : ex2((v - l) * LOG2E); };
                    gs[o] = g[u].x; gs[o + COL_LD] = g[u].y; gs[o + 2 * COL_LD] = g[u].z; gs[o + 3 * COL_LD] = g[u].w;
                    ps[o] = prob(x.x, ls[u].x); ps[o + COL_LD] = prob(x.y, ls[u].y);
                    ps[o + 2 * COL_LD] = prob(x.z, ls[u].z); ps[o + 3 * COL_LD] = prob(x.w, ls[u].w);
                }
                __syncthreads();
                if (i0 + COL_ROWS < n) fetch(i0 + COL_ROWS);
                const float *qp = p.q + (first + i0 + par) * HEADS * HEAD_DIM + h * HEAD_DIM + d;
                const float *gp = p.gout + (first + i0 + par) * HEADS * HEAD_DIM + h * HEAD_DIM + d;
                const float4 *g4 = reinterpret_cast<const float4 *>(gs + h * COL_LD + par * COL_KEYS);
                const float4 *p4 = reinterpret_cast<const float4 *>(ps + h * COL_LD + par * COL_KEYS);
                auto sum = [&](int u, float qv, float gv) {  // row 2u + par
                    const float4 g0 = g4[4 * u], g1 = g4[4 * u + 1], p0 = p4[4 * u], p1 = p4[4 * u + 1];
                    ak[0] = fmaf(g0.x, qv, ak[0]); ak[1] = fmaf(g0.y, qv, ak[1]); ak[2] = fmaf(g0.z, qv, ak[2]); ak[3] = fmaf(g0.w, qv, ak[3]);
                    ak[4] = fmaf(g1.x, qv, ak[4]); ak[5] = fmaf(g1.y, qv, ak[5]); ak[6] = fmaf(g1.z, qv, ak[6]); ak[7] = fmaf(g1.w, qv, ak[7]);
                    av[0] = fmaf(p0.x, gv, av[0]); av[1] = fmaf(p0.y, gv, av[1]); av[2] = fmaf(p0.z, gv, av[2]); av[3] = fmaf(p0.w, gv, av[3]);
                    av[4] = fmaf(p1.x, gv, av[4]); av[5] = fmaf(p1.y, gv, av[5]); av[6] = fmaf(p1.z, gv, av[6]); av[7] = fmaf(p1.w, gv, av[7]);
                };
                constexpr int STEP = 2 * HEADS * HEAD_DIM;
                int u0 = 0;
#pragma unroll
                for (int half = 0; half < 2; ++half) {  // sixteen rows at a time: constant offsets
                    if (rows < 16 * (half + 1)) break;
                    float qv[8], gv[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) { qv[u] = __ldg(qp + (8 * half + u) * STEP); gv[u] = __ldg(gp + (8 * half + u) * STEP); }
#pragma unroll
                    for (int u = 0; u < 8; ++u) sum(8 * half + u, qv[u], gv[u]);
                    u0 = 8 * (half + 1);
                }
#pragma unroll 4
                for (int u = u0; 2 * u + par < rows; ++u) sum(u, __ldg(qp + u * STEP), __ldg(gp + u * STEP));
            }
#pragma unroll
            for (int u = 0; u < COL_KEYS; ++u) {
                ak[u] += __shfl_xor_sync(FULL, ak[u], 16);
                av[u] += __shfl_xor_sync(FULL, av[u], 16);
                if (u < keys) (par == 0 ? p.gk : p.gv)[(j0 + u) * HEADS * HEAD_DIM + h * HEAD_DIM + d] = par == 0 ? ak[u] : av[u];
            }
            j0 += keys;
        }
    }
}

// LEFT: only the rows that a call over pair grids left over (p.rows_on_device of them), which also leave their probabilities
template <bool LEFT>
int launch_bwd(BwdRowArgs p, int64_t K, cudaStream_t s)
{
    p.pieces = (((uintptr_t)p.logit | (uintptr_t)p.lse | (uintptr_t)p.glogit | (uintptr_t)p.prob) & 15) == 0;
    const size_t smem = sizeof(float) * bwd_row_smem_floats(p.max_atoms, K > 0);
    const long long grid_rows = LEFT ? p.N / 8 + 1 : p.N;
    auto kernel = K > 0 ? infinite_attn_bwd_rows_kernel<64, LEFT> : infinite_attn_bwd_rows_kernel<0, LEFT>;
    if (smem > 48 * 1024) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return fail(CF_ERR_RANGE, "cf_infinite_attn_bwd: %zu bytes of shared memory for max_atoms=%d not available", smem, p.max_atoms);
        }
    }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, THREADS, smem) != cudaSuccess || occ <= 0) occ = 1;
    const long long cap = (long long)sm_count() * occ;
    kernel<<<(int)(grid_rows < cap ? grid_rows : cap), THREADS, smem, s>>>(p);
    const long long tiles = (p.N + COL_KEYS - 1) / COL_KEYS, cap2 = (long long)sm_count() * 8;
    infinite_attn_bwd_cols_kernel<LEFT><<<(int)(tiles < cap2 ? tiles : cap2), 256, 0, s>>>(p);
    return launch_status("cf_infinite_attn_bwd");
}

}  // namespace

int infinite_attn_bwd_impl(const float *q, const float *k, const float *v, const float *a, const float *pos,
                           const float *pos_ij, const float *tvecs, const float *rvlen, const int64_t *batch,
                           const int64_t *edges, const int64_t *row_start, int64_t N, int64_t B, int64_t H, int64_t D,
                           int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale, const float *W,
                           double cutoff_radius, int lattice_range, int minimum_range, const float *logit,
                           const float *lse, const float *out, const float *gout, float *gq, float *gk, float *gv,
                           float *ga, float *glogit, const int32_t *row_order, const TermList *list, void *stream);

// The backward over pair grids, by enumeration for the rows that the forward left over (p.leftover, counted in the grid's counters of
// the call), then the sums over the rows for k and v.
int grid_attn_bwd_impl(const PairAttn &l, const float *pos_ij, const float *tvecs, const int64_t *batch, const int64_t *edges,
                       const int64_t *row_start, cudaStream_t s)
{
    const int rc = launch_pair_attn_bwd(l, s);
    if (rc != CF_OK || l.N == 0) return rc;
    BwdRowArgs p{};
    p.q = l.q; p.k = l.k; p.v = l.v; p.a = l.a; p.pos_ij = pos_ij; p.tvecs = tvecs; p.rvlen = l.rvlen; p.W = l.W;
    p.logit = l.logit; p.lse = l.lse; p.out = l.out; p.gout = l.gout; p.batch = batch; p.edges = edges; p.row_start = row_start;
    p.gq = l.gq; p.gk = l.gk; p.gv = l.gv; p.ga = l.ga; p.glogit = l.glogit; p.prob = l.prob; p.N = l.N; p.E = l.E; p.max_atoms = l.max_atoms;
    p.row_order = l.leftover; p.rows_on_device = l.grid.counters + 4 * (l.call + 1);
    p.rule = l.rule;
    p.basis = make_basis_params(l.K, l.dist_max, l.wscale, weight_floor_log2());
    return launch_bwd<true>(p, l.K, s);
}

}  // namespace cf

extern "C" int cf_infinite_attn_bwd(const float *q, const float *k, const float *v, const float *a, const float *pos,
                                    const float *pos_ij, const float *tvecs, const float *rvlen, const int64_t *batch,
                                    const int64_t *edges, const int64_t *row_start, int64_t N, int64_t B, int64_t H,
                                    int64_t D, int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale,
                                    const float *W, double cutoff_radius, int lattice_range, int minimum_range,
                                    const float *logit, const float *lse, const float *out, const float *gout, float *gq,
                                    float *gk, float *gv, float *ga, float *glogit, const int32_t *row_order,
                                    void *stream)
{
    return cf::infinite_attn_bwd_impl(q, k, v, a, pos, pos_ij, tvecs, rvlen, batch, edges, row_start, N, B, H, D, E, K,
                                      max_atoms, dist_max, wscale, W, cutoff_radius, lattice_range, minimum_range, logit,
                                      lse, out, gout, gq, gk, gv, ga, glogit, row_order, nullptr, stream);
}

extern "C" int cf_infinite_attn_bwd_listed(const float *q, const float *k, const float *v, const float *a,
                                           const float *pos_ij, const float *tvecs, const float *rvlen,
                                           const int64_t *batch, const int64_t *edges, const int64_t *row_start,
                                           int64_t N, int64_t B, int64_t H, int64_t D, int64_t E, int64_t K,
                                           int64_t max_atoms, double dist_max, double wscale, const float *W,
                                           double cutoff_radius, int lattice_range, int minimum_range,
                                           const float *logit, const float *lse, const float *out, const float *gout,
                                           float *gq, float *gk, float *gv, float *ga, float *glogit,
                                           const int32_t *row_order, void *term_lists, double a_widest, void *stream)
{
    using namespace cf;
    CF_REQUIRE(term_lists != nullptr && pos_ij != nullptr && a_widest < 0, CF_ERR_INVALID,
               "cf_infinite_attn_bwd_listed: needs term lists, pos_ij and a negative a_widest");
    CF_REQUIRE(N >= 0 && E >= 0, CF_ERR_INVALID, "cf_infinite_attn_bwd_listed: negative size");
    TermList list{};
    int *start, *count;
    float *dmin;
    unsigned long long *cursor;
    float2 *pool;
    term_list_carve(term_lists, N, E, &start, &count, &dmin, &cursor, &pool);
    list.pool = pool; list.start = start; list.count = count; list.dmin = dmin;
    list.window = term_window(weight_floor_log2(), (float)a_widest);
    return infinite_attn_bwd_impl(q, k, v, a, nullptr, pos_ij, tvecs, rvlen, batch, edges, row_start, N, B, H, D, E, K,
                                  max_atoms, dist_max, wscale, W, cutoff_radius, lattice_range, minimum_range, logit, lse,
                                  out, gout, gq, gk, gv, ga, glogit, row_order, &list, stream);
}

int cf::infinite_attn_bwd_impl(const float *q, const float *k, const float *v, const float *a, const float *pos,
                               const float *pos_ij, const float *tvecs, const float *rvlen, const int64_t *batch,
                               const int64_t *edges, const int64_t *row_start, int64_t N, int64_t B, int64_t H,
                               int64_t D, int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale,
                               const float *W, double cutoff_radius, int lattice_range, int minimum_range,
                               const float *logit, const float *lse, const float *out, const float *gout, float *gq,
                               float *gk, float *gv, float *ga, float *glogit, const int32_t *row_order,
                               const TermList *list, void *stream)
{
    CF_REQUIRE(N >= 0 && E >= 0 && B >= 0, CF_ERR_INVALID, "cf_infinite_attn_bwd: negative size");
    CF_REQUIRE(H == HEADS && D == HEAD_DIM, CF_ERR_UNSUPPORTED, "cf_infinite_attn_bwd: H=%lld D=%lld, only H=8 D=16 is compiled",
               (long long)H, (long long)D);
    CF_REQUIRE(K == 0 || K == 64, CF_ERR_UNSUPPORTED, "cf_infinite_attn_bwd: K=%lld, only K in {0,64} is compiled", (long long)K);
    CF_REQUIRE(lattice_range >= 0 && lattice_range <= CF_MAX_RANGE && minimum_range >= 0, CF_ERR_RANGE,
               "cf_infinite_attn_bwd: lattice_range %d outside [0,%d]", lattice_range, CF_MAX_RANGE);
    CF_REQUIRE(max_atoms >= 1 && max_atoms <= 1024, CF_ERR_RANGE, "cf_infinite_attn_bwd: max_atoms=%lld outside [1,1024]",
               (long long)max_atoms);
    if (N == 0) return CF_OK;
    CF_REQUIRE(q && k && v && a && (pos || pos_ij) && tvecs && batch && edges && row_start && logit && lse && out && gout &&
                   gq && gk && gv && ga && glogit, CF_ERR_INVALID, "cf_infinite_attn_bwd: null pointer");
    CF_REQUIRE(K == 0 || (W != nullptr && dist_max > 0 && wscale > 0), CF_ERR_INVALID,
               "cf_infinite_attn_bwd: K > 0 needs W and positive dist_max, wscale");
    cudaStream_t s = as_stream(stream);
    BwdRowArgs p{};
    p.q = q; p.k = k; p.v = v; p.a = a; p.pos = pos; p.pos_ij = pos_ij; p.tvecs = tvecs; p.rvlen = rvlen; p.W = W;
    p.logit = logit; p.lse = lse; p.out = out; p.gout = gout; p.batch = batch; p.edges = edges; p.row_start = row_start;
    p.gq = gq; p.gk = gk; p.gv = gv; p.ga = ga; p.glogit = glogit; p.row_order = row_order; p.N = N; p.E = E; p.max_atoms = (int)max_atoms;
    p.rule = BoxRule{(float)cutoff_radius, lattice_range, minimum_range};
    p.basis = make_basis_params(K, dist_max, wscale, weight_floor_log2());
    if (list != nullptr) p.list = *list;
    return launch_bwd<false>(p, K, s);
}
