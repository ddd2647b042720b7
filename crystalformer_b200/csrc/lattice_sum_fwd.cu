// Real-space lattice sum, forward: phi (E,H) and psi (E,H,K) or W psi (E,H,16) per edge.
//
// lattice_edge_kernel: one warp per edge, phi and psi from one walk over the box (building blocks in lattice_edge.cuh and
// lattice_core.cuh).  The reference gives every (edge, head) its own thread and so repeats the geometry and the 64 basis
// exponentials eight times; here they are evaluated once per (edge, translation) and shared by the heads.
// lattice_phi_kernel: one thread per edge, phi alone; serves the fused attention where no term lists exist.
// The box of a head follows the reference rule exactly; heads of one edge may have different boxes, in which case
// the union box is enumerated and each head masks the translations outside its own.
#include "lattice_edge.cuh"

namespace cf {

namespace {

enum { AS_PSI = 0, ONE_W = 1, MANY_W = 2 };
constexpr int GROUP = 2;  // edges projected together: W is read from shared memory once for both
constexpr int PSI_STRIDE = 68;                            // floats per head row of the per-warp psi tile (bank skew)
constexpr int WT_HEAD_STRIDE = 64 * HEAD_DIM + 16;        // floats per head of the transposed projection (bank skew)

struct FwdArgs {
    const float *a;
    const float *pos_ij;
    const float *tvecs;
    const int64_t *batch;
    const int64_t *edges;
    const float *W;
    const float *rvlen;
    float *z;
    float *v;
    long long N, E, W_num;
    BoxRule rule;
    BasisParams basis;
    int a_per_edge;
};

// out[h][4 mq .. 4 mq + 3] = sum_k W[h][m][k] psi[h][k] for the lane's (h, mq), W in global memory, psi in shared memory.
template <int K>
__device__ __forceinline__ float4 project(const float *__restrict__ Wsrc, const float *__restrict__ psi, int lane)
{
    const int h = lane >> 2, mq = lane & 3;
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
    const float *ps = psi + h * PSI_STRIDE;
    const float *w = Wsrc + (size_t)(h * HEAD_DIM + 4 * mq) * K;  // [m][k]
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        const float4 pv = *reinterpret_cast<const float4 *>(ps + k);
        const float4 w0 = __ldg(reinterpret_cast<const float4 *>(w + 0 * K + k));
        const float4 w1 = __ldg(reinterpret_cast<const float4 *>(w + 1 * K + k));
        const float4 w2 = __ldg(reinterpret_cast<const float4 *>(w + 2 * K + k));
        const float4 w3 = __ldg(reinterpret_cast<const float4 *>(w + 3 * K + k));
        o0 += w0.x * pv.x + w0.y * pv.y + w0.z * pv.z + w0.w * pv.w;
        o1 += w1.x * pv.x + w1.y * pv.y + w1.z * pv.z + w1.w * pv.w;
        o2 += w2.x * pv.x + w2.y * pv.y + w2.z * pv.z + w2.w * pv.w;
        o3 += w3.x * pv.x + w3.y * pv.y + w3.z * pv.z + w3.w * pv.w;
    }
    return make_float4(o0, o1, o2, o3);
}

// The same for GROUP tiles at once with W staged as wt[h][k][m].
template <int K>
__device__ __forceinline__ void project_group(const float *__restrict__ wt_all, const float *__restrict__ psi, int lane, float4 (&o)[GROUP])
{
    const int h = lane >> 2, mq = lane & 3;
    const float *wt = wt_all + h * WT_HEAD_STRIDE + 4 * mq;
#pragma unroll
    for (int u = 0; u < GROUP; ++u) o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) w[t] = *reinterpret_cast<const float4 *>(wt + (k + t) * HEAD_DIM);
#pragma unroll
        for (int u = 0; u < GROUP; ++u) {
            const float4 pv = *reinterpret_cast<const float4 *>(psi + (u * 8 + h) * PSI_STRIDE + k);
            const float ps[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                o[u].x = fmaf(w[t].x, ps[t], o[u].x); o[u].y = fmaf(w[t].y, ps[t], o[u].y);
                o[u].z = fmaf(w[t].z, ps[t], o[u].z); o[u].w = fmaf(w[t].w, ps[t], o[u].w);
            }
        }
    }
}

template <int TPE>
__global__ void __launch_bounds__(128) lattice_phi_kernel(const PhiArgs p)
{
    const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gtid == 0 && p.zero_word) *p.zero_word = 0u;
    const long long e_raw = gtid / TPE;
    const int sub = (int)(gtid % TPE);
    const bool live = e_raw < p.E;
    const long long e = live ? e_raw : p.E - 1;  // idle tail threads shadow the last edge so that shuffles stay full
    const long long i = p.edges[e];
    const long long c = p.batch[i];
    Cell cell;
    cell.load(p.tvecs + 9 * c);
    const float4 *ap = reinterpret_cast<const float4 *>(p.a + (p.a_per_edge ? e : i) * HEADS);
    const float4 a_lo = __ldg(ap), a_hi = __ldg(ap + 1);
    const float a[8] = {a_lo.x, a_lo.y, a_lo.z, a_lo.w, a_hi.x, a_hi.y, a_hi.z, a_hi.w};
    float rx, ry, rz;
    if (p.pos_ij) {
        rx = p.pos_ij[3 * e]; ry = p.pos_ij[3 * e + 1]; rz = p.pos_ij[3 * e + 2];
    } else {
        const long long j = p.edges[p.E + e];
        rx = __fsub_rn(p.pos[3 * j], p.pos[3 * i]);
        ry = __fsub_rn(p.pos[3 * j + 1], p.pos[3 * i + 1]);
        rz = __fsub_rn(p.pos[3 * j + 2], p.pos[3 * i + 2]);
    }
    float z[8];
    edge_phi<TPE>(p.rule, a, p.rvlen ? p.rvlen + 3 * c : nullptr, cell, rx, ry, rz, p.floor_log2, sub, z);
    if (live && sub == 0) {
        float4 *zp = reinterpret_cast<float4 *>(p.z + e * HEADS);
        zp[0] = make_float4(z[0], z[1], z[2], z[3]);
        zp[1] = make_float4(z[4], z[5], z[6], z[7]);
    }
}

// One warp per edge: phi and, with K > 0, the radial-basis expansion (MODE: as psi; projected with one W staged in shared
// memory, four edges at a time; projected with a W per edge or atom).  Weights are taken relative to the nearest image,
//     w_n = exp(a (d2_n - m)),   phi = a m + log sum w_n,   psi = sum w_n g(d_n) / sum w_n,
// so one walk over the box gives both (an edge whose sum comes out empty - a head whose box misses the nearest image by
// far - is repeated with the normaliser of that head's own minimum).

// (the blocks that stage W have eight warps: 16 warps per SM then fit beside two copies of it)
__host__ __device__ constexpr int edge_warps(int mode) { return mode == ONE_W ? 8 : 4; }

template <int K, int MODE>
__global__ void __launch_bounds__(32 * edge_warps(MODE), K == 0 ? 6 : 16 / edge_warps(MODE)) lattice_edge_kernel(const FwdArgs p)
{
    constexpr int WARPS = edge_warps(MODE), THREADS = 32 * WARPS;
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int TILES = K == 0 ? 0 : MODE == ONE_W ? GROUP : 1;
    constexpr int WARP_FLOATS = EDGE_TERM_FLOATS + (K > 0 ? STAGE_FLOATS : 0) + TILES * 8 * PSI_STRIDE;
    float *wt = smem;
    float *mine = smem + (MODE == ONE_W ? HEADS * WT_HEAD_STRIDE : 0) + warp * WARP_FLOATS;
    float *psi = mine + EDGE_TERM_FLOATS + STAGE_FLOATS;
    if (MODE == ONE_W) {
        // W[h][m][k] -> wt[h][k][m] so that a lane reads its four outputs' weights as one float4
        for (int idx = threadIdx.x; idx < HEADS * HEAD_DIM * K; idx += THREADS) {
            const int h = idx / (HEAD_DIM * K), m = (idx / K) % HEAD_DIM, k = idx % K;
            wt[h * WT_HEAD_STRIDE + k * HEAD_DIM + m] = p.W[idx];
        }
        __syncthreads();
    }
    BinAccumulator<K> bins;
    if (K > 0) bins.init(mine + EDGE_TERM_FLOATS, lane, p.basis);
    EdgeTerms terms;
    terms.buf = reinterpret_cast<float2 *>(mine); terms.count = 0; terms.lane = lane;
    BoxWalk w5;
    w5.init(lane);
    EdgeStream es;
    es.a = p.a; es.pos_ij = p.pos_ij; es.tvecs = p.tvecs; es.rvlen = p.rvlen; es.batch = p.batch; es.edges = p.edges;
    es.E = p.E; es.a_per_edge = p.a_per_edge;
    const long long stride = (long long)gridDim.x * WARPS;
    es.begin((long long)blockIdx.x * WARPS + warp, stride, lane);
    long long group_e[GROUP];
    float group_inv[GROUP];
    int in_group = 0;

    for (; es.e < p.E; es.next()) {
        Cell cell;
        float rx, ry, rz, rvl[3];
        es.unpack(cell, rx, ry, rz, rvl);
        const float a_own = es.a_own;
        const int pk_own = packed_box(p.rule, a_own, p.rvlen ? rvl : nullptr);
        int uni = pk_own;
        float a2max = a_own;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            uni = box_union(uni, __shfl_xor_sync(FULL, uni, o));
            a2max = fmaxf(a2max, __shfl_xor_sync(FULL, a2max, o));
        }
        a2max *= LOG2E;
        const bool masked = !__all_sync(FULL, pk_own == uni);
        float a2[8];
        int pk[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            a2[h] = __shfl_sync(FULL, a_own, h) * LOG2E;
            pk[h] = __shfl_sync(FULL, pk_own, h) | 0x808080;
        }
        // ---- nearest image of the union box, then the terms whose largest weight is above the floor
        float S[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) S[h] = 0.f;
        if (K > 0) bins.clear();
        float m = fmaf(rz, rz, fmaf(ry, ry, rx * rx));
        auto weigh = [&](bool got, float d2, int key) {
            const float rel = d2 - m;
            float w[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                w[h] = ex2(a2[h] * rel);
                if (!got || (masked && !term_in_box(key, pk[h]))) w[h] = 0.f;
                S[h] += w[h];
            }
            if (K > 0) bins.push(got && d2 < p.basis.d2_cut, fast_sqrt(d2) * p.basis.bin_scale, w);
        };
        if (uni == BOX222) {
            float d2v[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                d2v[b] = term_d2(cell, rx, ry, rz, w5.f1[b], w5.f2[b], w5.f3[b]);
                if (b == 3 && lane >= 29) d2v[b] = INFINITY;
                m = fminf(m, d2v[b]);
            }
            m = warp_min(m);
#pragma unroll
            for (int b = 0; b < 4; ++b)
                terms.add(a2max * (d2v[b] - m) > p.basis.floor_log2, d2v[b], masked ? term_key(w5.f1[b], w5.f2[b], w5.f3[b]) : 0);
        } else {
            walk_box(w5, uni, cell, rx, ry, rz, lane,
                     [&](bool valid, float d2, float, float, float) { m = valid ? fminf(m, d2) : m; }, []() {});
            m = warp_min(m);
            walk_box(w5, uni, cell, rx, ry, rz, lane,
                     [&](bool valid, float d2, float f1, float f2, float f3) {
                         terms.add(valid && a2max * (d2 - m) > p.basis.floor_log2, d2, masked ? term_key(f1, f2, f3) : 0);
                     },
                     [&]() { if (terms.count >= 32) terms.consume(false, weigh); });
        }
        terms.consume(true, weigh);
        const int g = lane >> 2;
        const float S_g = warp_sum_of_8(S, lane), a_g = __shfl_sync(FULL, a_own, g);
        const int pk_g = __shfl_sync(FULL, pk_own, g);
        float z_g = fmaf(m, a_g, logf(S_g)), inv_g = __frcp_rn(S_g);
        if (__any_sync(FULL, !(S_g > 1e-30f))) {
            // a head's box misses the nearest image by hundreds of square Angstrom: phi from its own minimum, and the
            // expansion once more with normalised weights
            if (!(S_g > 1e-30f)) z_g = head_phi_own_min(cell, rx, ry, rz, a_g, pk_g);
            if (K > 0) {
                float off[8];
#pragma unroll
                for (int h = 0; h < 8; ++h) off[h] = -__shfl_sync(FULL, z_g, 4 * h) * LOG2E;
                bins.clear();
                auto again = [&](bool got, float d2, int key) {
                    float w[8], top = -INFINITY;
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        float eh = fmaf(a2[h], d2, off[h]);
                        if (!got || !term_in_box(key, pk[h])) eh = -INFINITY;
                        w[h] = ex2(eh);
                        top = fmaxf(top, eh);
                    }
                    bins.push(top > p.basis.floor_log2 && d2 < p.basis.d2_cut, fast_sqrt(d2) * p.basis.bin_scale, w);
                };
                walk_box(w5, uni, cell, rx, ry, rz, lane,
                         [&](bool valid, float d2, float f1, float f2, float f3) { terms.add(valid, d2, term_key(f1, f2, f3)); },
                         [&]() { if (terms.count >= 32) terms.consume(uni == BOX222, again); });
                terms.consume(true, again);
                inv_g = 1.0f;
            }
        }
        if ((lane & 3) == 0) p.z[es.e * HEADS + g] = z_g;
        if (K == 0) continue;
        if (MODE == AS_PSI) {
            bins.flush(psi, PSI_STRIDE);
            float4 *dst = reinterpret_cast<float4 *>(p.v + (size_t)es.e * HEADS * K) + lane;
#pragma unroll
            for (int t = 0; t < 4; ++t) {  // float4 lane + 32 t of the 8 x 64 block: head 2 t + lane / 16
                const int h = 2 * t + (lane >> 4);
                const float inv = __shfl_sync(FULL, inv_g, 4 * h);
                float4 v = *reinterpret_cast<const float4 *>(psi + h * PSI_STRIDE + 4 * (lane & 15));
                v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
                dst[32 * t] = v;
            }
            __syncwarp();
        } else if (MODE == MANY_W) {
            bins.flush(psi, PSI_STRIDE);
            const long long wi = p.W_num == p.E ? es.e : es.i;
            float4 o = project<K>(p.W + (size_t)wi * HEADS * HEAD_DIM * K, psi, lane);  // (lane = head lane / 4)
            o.x *= inv_g; o.y *= inv_g; o.z *= inv_g; o.w *= inv_g;
            reinterpret_cast<float4 *>(p.v + (size_t)es.e * HEADS * HEAD_DIM)[lane] = o;
            __syncwarp();
        } else {
            bins.flush(psi + in_group * 8 * PSI_STRIDE, PSI_STRIDE);
#pragma unroll
            for (int u = 0; u < GROUP; ++u)
                if (u == in_group) { group_e[u] = es.e; group_inv[u] = inv_g; }
            if (++in_group == GROUP || es.e + stride >= p.E) {
                float4 o[GROUP];
                project_group<K>(wt, psi, lane, o);
#pragma unroll
                for (int u = 0; u < GROUP; ++u)
                    if (u < in_group)
                        reinterpret_cast<float4 *>(p.v + (size_t)group_e[u] * HEADS * HEAD_DIM)[lane] =
                            make_float4(o[u].x * group_inv[u], o[u].y * group_inv[u], o[u].z * group_inv[u], o[u].w * group_inv[u]);
                in_group = 0;
                __syncwarp();
            }
        }
    }
}

__global__ void lattice_box_kernel(const float *a, int a_per_edge, const int64_t *batch, const int64_t *edges,
                                   long long E, const float *rvlen, BoxRule rule, int32_t *box)
{
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= E * HEADS) return;
    const long long e = tid / HEADS;
    const int h = (int)(tid % HEADS);
    const long long i = edges[e];
    const long long c = batch[i];
    // the very function the lattice-sum kernels call, so that the bit-exactness test covers what they enumerate
    const int pk = packed_box(rule, a[(a_per_edge ? e : i) * HEADS + h], rvlen ? rvlen + 3 * c : nullptr);
    box[3 * tid + 0] = box_r1(pk);
    box[3 * tid + 1] = box_r2(pk);
    box[3 * tid + 2] = box_r3(pk);
}


int launch_fwd(const FwdArgs &p, long long K, cudaStream_t stream)
{
    const int mode = K == 0 ? 3 : p.W == nullptr ? AS_PSI : p.W_num == 1 ? ONE_W : MANY_W;
    void (*const kernels[4])(const FwdArgs) = {lattice_edge_kernel<64, AS_PSI>, lattice_edge_kernel<64, ONE_W>,
                                               lattice_edge_kernel<64, MANY_W>, lattice_edge_kernel<0, AS_PSI>};
    const int warps = edge_warps(mode), threads = 32 * warps;
    const int tiles = mode == 3 ? 0 : mode == ONE_W ? GROUP : 1;
    const size_t smem = sizeof(float) * ((mode == ONE_W ? HEADS * WT_HEAD_STRIDE : 0) +
                                         warps * (EDGE_TERM_FLOATS + (K > 0 ? STAGE_FLOATS : 0) + tiles * 8 * PSI_STRIDE));
    static thread_local int per_sm[4] = {0, 0, 0, 0};
    int &occ = per_sm[mode];
    if (occ == 0) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(kernels[mode], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernels[mode], threads, smem) != cudaSuccess || occ <= 0) occ = 2;
    }
    const long long want = (p.E + warps - 1) / warps;
    const long long cap = (long long)sm_count() * occ;
    kernels[mode]<<<(int)(want < cap ? want : cap), threads, smem, stream>>>(p);
    return launch_status("cf_lattice_sum_fwd");
}

}  // namespace

int launch_lattice_phi(const PhiArgs &p, cudaStream_t stream)
{
    if (p.E > 0) {
        // enough threads to give every SM about 24 warps: small batches split each edge over up to 8 threads
        const long long target = (long long)sm_count() * 24 * 32;
        int tpe = 1;
        while (tpe < 8 && p.E * tpe < target) tpe *= 2;
        const unsigned blocks = (unsigned)((p.E * tpe + 127) / 128);
        switch (tpe) {
            case 1: lattice_phi_kernel<1><<<blocks, 128, 0, stream>>>(p); break;
            case 2: lattice_phi_kernel<2><<<blocks, 128, 0, stream>>>(p); break;
            case 4: lattice_phi_kernel<4><<<blocks, 128, 0, stream>>>(p); break;
            default: lattice_phi_kernel<8><<<blocks, 128, 0, stream>>>(p); break;
        }
    }
    return launch_status("lattice_phi_kernel");
}

}  // namespace cf

extern "C" int cf_lattice_box(const float *a, int a_per_edge, const int64_t *batch, const int64_t *edges, int64_t N,
                              int64_t H, int64_t E, const float *rvlen, double cutoff_radius, int lattice_range,
                              int minimum_range, int32_t *box, void *stream)
{
    using namespace cf;
    CF_REQUIRE(N >= 0 && E >= 0, CF_ERR_INVALID, "cf_lattice_box: negative size");
    CF_REQUIRE(H == HEADS, CF_ERR_UNSUPPORTED, "cf_lattice_box: H=%lld, only H=8 is compiled", (long long)H);
    CF_REQUIRE(lattice_range >= 0 && lattice_range <= CF_MAX_RANGE && minimum_range >= 0, CF_ERR_RANGE,
               "cf_lattice_box: lattice_range %d outside [0,%d]", lattice_range, CF_MAX_RANGE);
    if (E == 0) return CF_OK;
    CF_REQUIRE(a && batch && edges && box, CF_ERR_INVALID, "cf_lattice_box: null pointer");
    BoxRule rule{(float)cutoff_radius, lattice_range, minimum_range};
    const long long total = (long long)E * HEADS;
    lattice_box_kernel<<<(unsigned)((total + 255) / 256), 256, 0, as_stream(stream)>>>(a, a_per_edge, batch, edges, E, rvlen, rule, box);
    return launch_status("cf_lattice_box");
}

extern "C" int cf_lattice_sum_fwd(const float *a, int a_per_edge, const float *pos_ij, const float *tvecs,
                                  const int64_t *batch, const int64_t *edges, int64_t N, int64_t H, int64_t E,
                                  int64_t K, double dist_max, double wscale, const float *W, int64_t W_num, int64_t Dv,
                                  const float *rvlen, double cutoff_radius, int lattice_range, int minimum_range,
                                  float *z, float *v, void *stream)
{
    using namespace cf;
    CF_REQUIRE(N >= 0 && E >= 0, CF_ERR_INVALID, "cf_lattice_sum_fwd: negative size");
    CF_REQUIRE(H == HEADS, CF_ERR_UNSUPPORTED, "cf_lattice_sum_fwd: H=%lld, only H=8 is compiled", (long long)H);
    CF_REQUIRE(K == 0 || K == 64, CF_ERR_UNSUPPORTED, "cf_lattice_sum_fwd: K=%lld, only K in {0,64} is compiled", (long long)K);
    CF_REQUIRE(lattice_range >= 0 && lattice_range <= CF_MAX_RANGE && minimum_range >= 0, CF_ERR_RANGE,
               "cf_lattice_sum_fwd: lattice_range %d outside [0,%d]", lattice_range, CF_MAX_RANGE);
    if (E == 0) return CF_OK;
    CF_REQUIRE(a && pos_ij && tvecs && batch && edges && z, CF_ERR_INVALID, "cf_lattice_sum_fwd: null pointer");
    if (K > 0) {
        CF_REQUIRE(v != nullptr, CF_ERR_INVALID, "cf_lattice_sum_fwd: v is null but K > 0");
        CF_REQUIRE(dist_max > 0 && wscale > 0, CF_ERR_INVALID, "cf_lattice_sum_fwd: dist_max and wscale must be positive");
        if (W) {
            CF_REQUIRE(Dv == HEAD_DIM, CF_ERR_UNSUPPORTED, "cf_lattice_sum_fwd: Dv=%lld, only 16 is compiled", (long long)Dv);
            CF_REQUIRE(W_num == 1 || W_num == E || W_num == N, CF_ERR_INVALID,
                       "cf_lattice_sum_fwd: W_num=%lld must be 1, E or N", (long long)W_num);
        }
    }
    FwdArgs p{};
    p.a = a; p.pos_ij = pos_ij; p.tvecs = tvecs; p.batch = batch; p.edges = edges;
    p.W = (K > 0) ? W : nullptr; p.rvlen = rvlen; p.z = z; p.v = v;
    p.N = N; p.E = E; p.W_num = W_num;
    p.rule = BoxRule{(float)cutoff_radius, lattice_range, minimum_range};
    p.a_per_edge = a_per_edge;
    p.basis = make_basis_params(K, dist_max, wscale, weight_floor_log2());
    return launch_fwd(p, K, as_stream(stream));
}
