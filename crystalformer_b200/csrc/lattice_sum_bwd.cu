// Real-space lattice sum, backward with respect to the Gaussian parameter a (N,H).
//
// Per edge e = (i,j) and head h, with p_n = exp(a d2_n - z_e) (z from the forward) and c_n = sum_k u_e[k] g_k(d_n)
// (u = gradient arriving at psi_e):
//     C0 = sum_n p_n c_n,  C1 = sum_n p_n d2_n,  C2 = sum_n p_n d2_n c_n
//     d loss / d a_i  +=  gz_e C1 + C2 - C1 C0
// (the formula of models/kernels/real_enc_bwd.cu:80-156).  One warp owns one edge (lattice_edge.cuh): the terms within
// reach are collected first, then every lane takes one of them, for the sums and for psi alike.
// The per-edge contributions are written out and summed per source atom by a second kernel in edge order, so the
// result does not depend on scheduling.  Optionally psi_e itself is recomputed and written (the gradient of a
// projection W needs it); phi and psi are never stored by the forward.
#include "lattice_bwd_core.cuh"
#include "lattice_edge.cuh"

namespace cf {
namespace {

constexpr int THREADS = 128;
constexpr int WARPS = THREADS / 32;
constexpr int KBINS = 64;
constexpr int PSI_STRIDE = 68;  // floats per head row of the psi tile (bank skew)
constexpr int WARP_SMEM_FLOATS = EDGE_TERM_FLOATS + HEADS * U_STRIDE + HEADS * PSI_STRIDE + STAGE_FLOATS;

struct BwdArgs {
    const float *a, *pos_ij, *tvecs, *rvlen, *z, *gz, *gpsi;
    const int64_t *batch, *edges;
    float *edge_out, *psi_out;
    long long E;
    BoxRule rule;
    BasisParams basis;
};

template <int K>
__global__ void __launch_bounds__(THREADS, 4) lattice_bwd_edges_kernel(const BwdArgs p)
{
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *mine = smem + warp * (K > 0 ? WARP_SMEM_FLOATS : EDGE_TERM_FLOATS);
    float *u = mine + EDGE_TERM_FLOATS;
    float *tile = u + HEADS * U_STRIDE;      // per-bin totals of the recomputed psi
    float *stage = tile + HEADS * PSI_STRIDE;
    BinAccumulator<KBINS> bins;
    if (K > 0) bins.init(stage, lane, p.basis);
    EdgeTerms terms;
    terms.buf = reinterpret_cast<float2 *>(mine); terms.count = 0; terms.lane = lane;
    BoxWalk w5;
    w5.init(lane);
    EdgeStream es;
    es.a = p.a; es.pos_ij = p.pos_ij; es.tvecs = p.tvecs; es.rvlen = p.rvlen; es.batch = p.batch; es.edges = p.edges;
    es.E = p.E; es.a_per_edge = 0;
    const bool with_u = K > 0 && p.gpsi != nullptr, with_psi = K > 0 && p.psi_out != nullptr;
    const int g = lane >> 2;

    for (es.begin((long long)blockIdx.x * WARPS + warp, (long long)gridDim.x * WARPS, lane); es.e < p.E; es.next()) {
        const long long e = es.e;
        if (with_u) {  // the edge's u arrives while the box is walked
            const unsigned dst = (unsigned)__cvta_generic_to_shared(u) + 16u * lane;
            const float *src = p.gpsi + (size_t)e * HEADS * K + 4 * lane;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512u * t), "l"(src + 128 * t));
            asm volatile("cp.async.commit_group;");
        }
        const float z_own = p.z[e * HEADS + (lane & 7)], gz_g = p.gz[e * HEADS + g];
        Cell cell;
        float rx, ry, rz, rvl[3];
        es.unpack(cell, rx, ry, rz, rvl);
        const float a_own = es.a_own, off_own = -z_own * LOG2E;
        const int pk_own = packed_box(p.rule, a_own, p.rvlen ? rvl : nullptr);
        int uni = pk_own;
        float a2max = a_own, off_max = off_own;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            uni = box_union(uni, __shfl_xor_sync(FULL, uni, o));
            a2max = fmaxf(a2max, __shfl_xor_sync(FULL, a2max, o));
            off_max = fmaxf(off_max, __shfl_xor_sync(FULL, off_max, o));
        }
        a2max *= LOG2E;
        const bool masked = !__all_sync(FULL, pk_own == uni);
        float a2[8], off[8];
        int pk[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            a2[h] = __shfl_sync(FULL, a_own, h) * LOG2E;
            off[h] = __shfl_sync(FULL, off_own, h);
            pk[h] = __shfl_sync(FULL, pk_own, h) | 0x808080;
        }
        float C0[8], C1[8], C2[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) C0[h] = C1[h] = C2[h] = 0.f;
        if (with_psi) bins.clear();
        auto weigh = [&](bool got, float d2, int key) {
            float w[8], top = -INFINITY;
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                float eh = fmaf(a2[h], d2, off[h]);
                if (!got || (masked && !term_in_box(key, pk[h]))) eh = -INFINITY;
                w[h] = ex2(eh);
                top = fmaxf(top, eh);
                C1[h] = fmaf(w[h], d2, C1[h]);
            }
            if (K > 0) {
                const float x = fast_sqrt(d2) * p.basis.bin_scale;
                const bool keep = top > p.basis.floor_log2 && d2 < p.basis.d2_cut;
                if (with_psi) bins.push(keep, x, w);
                if (with_u && keep) {
                    float cd[8];
                    if (K == 64 && p.basis.windowed) basis_dot_window(u, x, p.basis.bin_step, cd);
                    else basis_dot<(K > 0 ? K : 4)>(u, x, p.basis.bin_step, cd);
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        const float pc = w[h] * cd[h];
                        C0[h] += pc;
                        C2[h] = fmaf(pc, d2, C2[h]);
                    }
                }
                __syncwarp();
            }
        };
        // terms that some head's weight could bring above the floor
        auto reach = [&](float d2) { return fmaf(a2max, d2, off_max) > p.basis.floor_log2; };
        if (with_u) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
        }
        walk_box(w5, uni, cell, rx, ry, rz, lane,
                 [&](bool valid, float d2, float f1, float f2, float f3) {
                     terms.add(valid && reach(d2), d2, masked ? term_key(f1, f2, f3) : 0);
                 },
                 [&]() { if (terms.count >= 32) terms.consume(uni == BOX222, weigh); });
        terms.consume(true, weigh);
        if (with_psi) {
            bins.flush(tile, PSI_STRIDE);
            float4 *dst = reinterpret_cast<float4 *>(p.psi_out + (size_t)e * HEADS * KBINS) + lane;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                dst[32 * t] = *reinterpret_cast<const float4 *>(tile + (2 * t + (lane >> 4)) * PSI_STRIDE + 4 * (lane & 15));
        }
        const float c0 = warp_sum_of_8(C0, lane), c1 = warp_sum_of_8(C1, lane), c2 = warp_sum_of_8(C2, lane);
        if ((lane & 3) == 0) p.edge_out[e * HEADS + g] = fmaf(gz_g, c1, c2 - c1 * c0);
        __syncwarp();
    }
}

// ga[i][h] = sum of the contributions of atom i's edges, in edge order.
__global__ void row_sum_kernel(const float *__restrict__ edge_out, const int64_t *__restrict__ row_start, long long N,
                               float *__restrict__ ga)
{
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= N * HEADS) return;
    const long long i = tid / HEADS;
    const int h = (int)(tid % HEADS);
    float s = 0.f;
    for (long long e = row_start[i]; e < row_start[i + 1]; ++e) s += edge_out[e * HEADS + h];
    ga[tid] = s;
}

// gpsi[e][h][k] = sum_m W[h][m][k] gv[e][h][m]: thread = (head, bin) with its sixteen weights in registers, edges sixteen at
// a time through shared memory (broadcast reads).  Writes 2 KB per edge and is bound by that.
constexpr int UP_ROWS = 16;
__global__ void __launch_bounds__(512) project_back_kernel(const float *__restrict__ gv, const float *__restrict__ W, long long E,
                                                           float *__restrict__ gpsi)
{
    __shared__ __align__(16) float go[UP_ROWS * HEADS * HEAD_DIM];
    const int tid = threadIdx.x, h = tid >> 6, k = tid & 63;
    float w[HEAD_DIM];
#pragma unroll
    for (int m = 0; m < HEAD_DIM; ++m) w[m] = W[(h * HEAD_DIM + m) * KBINS + k];
    for (long long e0 = (long long)blockIdx.x * UP_ROWS; e0 < E; e0 += (long long)gridDim.x * UP_ROWS) {
        const int rows = (int)min((long long)UP_ROWS, E - e0);
        __syncthreads();
        const float *src = gv + e0 * HEADS * HEAD_DIM;
        if ((reinterpret_cast<uintptr_t>(gv) & 15) == 0) {
            for (int i = tid; i < rows * 32; i += 512) reinterpret_cast<float4 *>(go)[i] = __ldg(reinterpret_cast<const float4 *>(src) + i);
        } else {  // (a view into something longer)
            for (int i = tid; i < rows * 128; i += 512) go[i] = __ldg(src + i);
        }
        __syncthreads();
#pragma unroll 4
        for (int r = 0; r < rows; ++r) {
            const float4 *g4 = reinterpret_cast<const float4 *>(go + r * HEADS * HEAD_DIM + h * HEAD_DIM);
            float t0 = 0.f, t1 = 0.f;
#pragma unroll
            for (int m = 0; m < 4; m += 2) {
                const float4 x = g4[m], y = g4[m + 1];
                t0 = fmaf(x.x, w[4 * m], t0); t0 = fmaf(x.y, w[4 * m + 1], t0); t0 = fmaf(x.z, w[4 * m + 2], t0); t0 = fmaf(x.w, w[4 * m + 3], t0);
                t1 = fmaf(y.x, w[4 * m + 4], t1); t1 = fmaf(y.y, w[4 * m + 5], t1); t1 = fmaf(y.z, w[4 * m + 6], t1); t1 = fmaf(y.w, w[4 * m + 7], t1);
            }
            gpsi[(e0 + r) * 512 + tid] = t0 + t1;
        }
    }
}

}  // namespace
size_t projection_grad_floats(long long rows);
int launch_projection_grad(const float *gv, const float *psi, long long rows, float *gW, float *partial, cudaStream_t s);
}  // namespace cf

extern "C" int64_t cf_lattice_sum_bwd_proj_floats(int64_t E)
{
    return E > 0 ? (int64_t)(E * 8 + 2 * E * 512 + (int64_t)cf::projection_grad_floats(E)) : 8;
}

extern "C" int cf_lattice_sum_bwd_proj(const float *a, const float *pos_ij, const float *tvecs, const int64_t *batch,
                                       const int64_t *edges, const int64_t *row_start, const float *z, const float *gz,
                                       const float *gv, const float *W, int64_t N, int64_t H, int64_t E, int64_t K, double dist_max,
                                       double wscale, const float *rvlen, double cutoff_radius, int lattice_range,
                                       int minimum_range, float *ga, float *gW, float *workspace, void *stream)
{
    using namespace cf;
    CF_REQUIRE(N >= 0 && E >= 0, CF_ERR_INVALID, "cf_lattice_sum_bwd_proj: negative size");
    CF_REQUIRE(H == HEADS && K == KBINS, CF_ERR_UNSUPPORTED, "cf_lattice_sum_bwd_proj: H=%lld K=%lld, only H=8 K=64 is compiled",
               (long long)H, (long long)K);
    CF_REQUIRE(gW && (E == 0 || (gv && W && workspace)), CF_ERR_INVALID, "cf_lattice_sum_bwd_proj: null pointer");
    cudaStream_t s = as_stream(stream);
    if (E == 0 && cudaMemsetAsync(gW, 0, sizeof(float) * HEADS * HEAD_DIM * KBINS, s) != cudaSuccess) return launch_status("cf_lattice_sum_bwd_proj");
    float *gpsi = workspace, *psi = gpsi + E * 512, *scratch = psi + E * 512, *partial = scratch + E * 8;
    if (E > 0) {
        const long long want = (E + UP_ROWS - 1) / UP_ROWS, cap = 2ll * sm_count();
        project_back_kernel<<<(unsigned)(want < cap ? want : cap), 512, 0, s>>>(gv, W, E, gpsi);
    }
    int rc = cf_lattice_sum_bwd(a, pos_ij, tvecs, batch, edges, row_start, z, gz, gpsi, N, H, E, K, dist_max, wscale, rvlen, cutoff_radius,
                                lattice_range, minimum_range, ga, psi, scratch, stream);
    if (rc == CF_OK && E > 0) rc = launch_projection_grad(gv, psi, E, gW, partial, s);
    return rc;
}

extern "C" int cf_lattice_sum_bwd(const float *a, const float *pos_ij, const float *tvecs, const int64_t *batch,
                                  const int64_t *edges, const int64_t *row_start, const float *z, const float *gz,
                                  const float *gpsi, int64_t N, int64_t H, int64_t E, int64_t K, double dist_max,
                                  double wscale, const float *rvlen, double cutoff_radius, int lattice_range,
                                  int minimum_range, float *ga, float *psi_out, float *edge_scratch, void *stream)
{
    using namespace cf;
    CF_REQUIRE(N >= 0 && E >= 0, CF_ERR_INVALID, "cf_lattice_sum_bwd: negative size");
    CF_REQUIRE(H == HEADS, CF_ERR_UNSUPPORTED, "cf_lattice_sum_bwd: H=%lld, only H=8 is compiled", (long long)H);
    CF_REQUIRE(K == 0 || K == 64, CF_ERR_UNSUPPORTED, "cf_lattice_sum_bwd: K=%lld, only K in {0,64} is compiled", (long long)K);
    CF_REQUIRE(lattice_range >= 0 && lattice_range <= CF_MAX_RANGE && minimum_range >= 0, CF_ERR_RANGE,
               "cf_lattice_sum_bwd: lattice_range %d outside [0,%d]", lattice_range, CF_MAX_RANGE);
    if (N == 0) return CF_OK;
    CF_REQUIRE(ga && row_start, CF_ERR_INVALID, "cf_lattice_sum_bwd: null pointer");
    cudaStream_t s = as_stream(stream);
    if (E > 0) {
        CF_REQUIRE(a && pos_ij && tvecs && batch && edges && z && gz && edge_scratch, CF_ERR_INVALID,
                   "cf_lattice_sum_bwd: null pointer");
        CF_REQUIRE(K == 0 || (dist_max > 0 && wscale > 0), CF_ERR_INVALID, "cf_lattice_sum_bwd: dist_max and wscale must be positive");
        BwdArgs p{};
        p.a = a; p.pos_ij = pos_ij; p.tvecs = tvecs; p.rvlen = rvlen; p.z = z; p.gz = gz; p.gpsi = K > 0 ? gpsi : nullptr;
        p.batch = batch; p.edges = edges; p.edge_out = edge_scratch; p.psi_out = K > 0 ? psi_out : nullptr; p.E = E;
        p.rule = BoxRule{(float)cutoff_radius, lattice_range, minimum_range};
        p.basis = make_basis_params(K, dist_max, wscale, weight_floor_log2());
        const size_t smem = sizeof(float) * WARPS * (K > 0 ? WARP_SMEM_FLOATS : EDGE_TERM_FLOATS);
        const long long want = (E + WARPS - 1) / WARPS, cap = (long long)sm_count() * 4;
        const int blocks = (int)(want < cap ? want : cap);
        if (K > 0) lattice_bwd_edges_kernel<64><<<blocks, THREADS, smem, s>>>(p);
        else lattice_bwd_edges_kernel<0><<<blocks, THREADS, smem, s>>>(p);
    }
    const long long total = (long long)N * HEADS;
    row_sum_kernel<<<(unsigned)((total + 127) / 128), 128, 0, s>>>(edge_scratch, row_start, N, ga);
    return launch_status("cf_lattice_sum_bwd");
}

// ------------------------------------------------------------------------------------------------------------------
// cf_lattice_sum_bwd_static: the same computation for callers that cannot hand over a scratch buffer.
//
// Some embedders are not in a position to allocate device memory at the moment they call: a serving process that
// sized all of its device memory at start-up and gives libraries none afterwards, a binding from a language runtime
// that has no device allocator at hand, or a latency-critical loop in which an allocation (which may synchronise the
// whole device) is not acceptable.  For them the per-edge contributions live in a fixed array that is part of the
// library image itself: it costs CF_STATIC_SCRATCH_MAX_EDGES * 8 floats (8 MiB) on every GPU that loads the library,
// for as long as the process lives, and bounds the number of edges one call may have.
//
// The array's name is only meaningful to device code; host code must ask the runtime for its device address.  That
// is done once per device, on the first call made with that device current (so make the first call on each device
// outside any stream capture), and the address is remembered.  Every call on a device uses the same array: two calls
// whose kernels may overlap on the GPU (different streams) would overwrite each other's contributions, so callers
// must serialise them.  Nothing in the array needs clearing between calls: every element a call reads (edges
// 0..E-1) is written by that same call first.
// ------------------------------------------------------------------------------------------------------------------
#include <mutex>

static __device__ __align__(256) float g_static_edge_scratch[(size_t)CF_STATIC_SCRATCH_MAX_EDGES * 8];

extern "C" int cf_lattice_sum_bwd_static(const float *a, const float *pos_ij, const float *tvecs, const int64_t *batch,
                                         const int64_t *edges, const int64_t *row_start, const float *z,
                                         const float *gz, const float *gpsi, int64_t N, int64_t H, int64_t E, int64_t K,
                                         double dist_max, double wscale, const float *rvlen, double cutoff_radius,
                                         int lattice_range, int minimum_range, float *ga, float *psi_out, void *stream)
{
    using namespace cf;
    CF_REQUIRE(E <= (int64_t)CF_STATIC_SCRATCH_MAX_EDGES, CF_ERR_RANGE,
               "cf_lattice_sum_bwd_static: E=%lld exceeds the built-in scratch of %lld edges; use cf_lattice_sum_bwd "
               "with a caller-provided scratch buffer", (long long)E, (long long)CF_STATIC_SCRATCH_MAX_EDGES);
    constexpr int MAX_DEVICES = 64;
    static std::mutex lock;
    static float *address_on_device[MAX_DEVICES] = {};
    int dev = -1;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess || dev < 0 || dev >= MAX_DEVICES)
        return fail(CF_ERR_CUDA, "cf_lattice_sum_bwd_static: cudaGetDevice: %s", cudaGetErrorString(err));
    float *scratch = nullptr;
    {
        std::lock_guard<std::mutex> guard(lock);
        if (address_on_device[dev] == nullptr) {
            float *ptr = nullptr;
            err = cudaGetSymbolAddress((void **)&ptr, g_static_edge_scratch);
            if (err != cudaSuccess || ptr == nullptr) {
                cudaGetLastError();
                return fail(CF_ERR_CUDA, "cf_lattice_sum_bwd_static: cudaGetSymbolAddress: %s", cudaGetErrorString(err));
            }
            address_on_device[dev] = ptr;
        }
        scratch = address_on_device[dev];
    }
    return cf_lattice_sum_bwd(a, pos_ij, tvecs, batch, edges, row_start, z, gz, gpsi, N, H, E, K, dist_max, wscale, rvlen,
                              cutoff_radius, lattice_range, minimum_range, ga, psi_out, scratch, stream);
}
