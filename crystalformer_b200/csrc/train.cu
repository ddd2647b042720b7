// One training step of the whole model in two host calls: the forward (keeping what the backward needs) and the backward
// (gradients of every parameter).
//
// The autograd path records some sixty framework operations per layer; on a batch of crystals each of them is a few
// microseconds of device work, and the host needs about 5 ms to issue them.  Here a step is about forty launches of this
// library's kernels:
//   forward    weight images (both directions), batch geometry, pair grids or term lists, then per layer the dense boundary
//              (dense_tc.cu) and the fused attention (pair_attn.cu or infinite_attn_fwd.cu), pooling + head
//   backward   head and pooling, then per layer the dense boundary (dense_tc_bwd.cu) and the attention backward
//              (pair_attn_bwd.cu, infinite_attn_bwd.cu), and at the end every weight gradient of the model in one launch each for the
//              projections and for the value encoding
// (models/latticeformer.py:211-302 with pooling "avr", a Linear - ReLU - Linear head and LayerNorm = Identity.)
#include "common.cuh"
#include "dense_tc.cuh"
#include "infinite_attn_block.cuh"
#include "pair_grid.cuh"
#include "term_list.cuh"

namespace cf {
cudaStream_t early_prep_stream(void *inputs_ready, void *slot_free);
int join_early_prep(cudaStream_t s);
int launch_prepare_all(const float *pos, const float *trans, const int64_t *sizes, int64_t *atom_start,
                       int64_t *edge_start, long long B, long long N, long long E, int64_t *batch, int64_t *edges,
                       int64_t *row_start, float *pos_ij, float *rvlen, double reach, int32_t *row_order, bool *ordered,
                       cudaStream_t s, float *rvecs = nullptr, float *vcell = nullptr);
int infinite_attn_fwd_impl(const float *q, const float *k, const float *v, const float *a, const float *pos,
                           const float *pos_ij, const float *tvecs, const float *rvlen, const int64_t *batch,
                           const int64_t *edges, const int64_t *row_start, int64_t N, int64_t B, int64_t H, int64_t D,
                           int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale, const float *W,
                           double cutoff_radius, int lattice_range, int minimum_range, float *out, float *logit,
                           float *lse, float *psi_row, const int32_t *row_order, const TermList *list,
                           unsigned *ticket_ready, void *stream, bool chained);
int infinite_attn_bwd_impl(const float *q, const float *k, const float *v, const float *a, const float *pos,
                           const float *pos_ij, const float *tvecs, const float *rvlen, const int64_t *batch,
                           const int64_t *edges, const int64_t *row_start, int64_t N, int64_t B, int64_t H, int64_t D,
                           int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale, const float *W,
                           double cutoff_radius, int lattice_range, int minimum_range, const float *logit,
                           const float *lse, const float *out, const float *gout, float *gq, float *gk, float *gv,
                           float *ga, float *glogit, const int32_t *row_order, const TermList *list, void *stream);
int launch_pool_head(const float *x, const int64_t *atom_start, const float *W1, const float *b1, const float *W2,
                     const float *b2, int hidden, int targets, long long B, float *y, float *pooled, float *hid, bool chained,
                     cudaStream_t s);
namespace {

constexpr int CH = HEADS * HEAD_DIM;  // 128

// ---- head and pooling, backward: one block per crystal ------------------------------------------------------------------
__global__ void __launch_bounds__(128) head_backward_kernel(const float *__restrict__ gy, const float *__restrict__ hid,
                                                            const float *__restrict__ W1, const float *__restrict__ W2,
                                                            const int64_t *__restrict__ atom_start, int hidden, int targets,
                                                            float *__restrict__ ghid, float *__restrict__ gx)
{
    __shared__ float gh[1024];
    const long long c = blockIdx.x;
    const int tid = threadIdx.x;
    for (int u = tid; u < hidden; u += 128) {
        float g = 0.f;
        for (int t = 0; t < targets; ++t) g = fmaf(gy[c * targets + t], __ldg(W2 + (size_t)t * hidden + u), g);
        g = hid[c * hidden + u] > 0.f ? g : 0.f;
        gh[u] = g;
        ghid[c * hidden + u] = g;
    }
    __syncthreads();
    float g0 = 0.f, g1 = 0.f;
#pragma unroll 8
    for (int u = 0; u < hidden; u += 2) {
        g0 = fmaf(gh[u], __ldg(W1 + (size_t)u * CH + tid), g0);
        g1 = fmaf(gh[u + 1], __ldg(W1 + (size_t)(u + 1) * CH + tid), g1);
    }
    const long long s = atom_start[c], n = atom_start[c + 1] - s;
    const float g = (g0 + g1) / (float)n;
    for (long long r = 0; r < n; ++r) gx[(s + r) * CH + tid] = g;
}

// gradient of the head's last layer: gW2[t][u] = sum_c gy[c][t] hid[c][u], gb2[t] = sum_c gy[c][t].  Block = (32 units,
// target); the warps take every eighth crystal (compensated sums: a batch may have thousands) and meet in shared memory in a
// fixed order.
__global__ void __launch_bounds__(256) head_weight_grad_kernel(const float *__restrict__ gy, const float *__restrict__ hid, long long B,
                                                               int hidden, int targets, float *__restrict__ gW2, float *__restrict__ gb2)
{
    __shared__ float part[2][8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, u = blockIdx.x * 32 + lane, t = blockIdx.y;
    float acc = 0.f, acc_low = 0.f, bias = 0.f, bias_low = 0.f;
    for (long long c = w; c < B; c += 8) {
        const float g = gy[c * targets + t];
        add_compensated(g * (u < hidden ? hid[c * hidden + u] : 0.f), acc, acc_low);
        add_compensated(g, bias, bias_low);
    }
    part[0][w][lane] = acc + acc_low;
    part[1][w][lane] = bias + bias_low;
    __syncthreads();
    if (w == 0) {
        auto eight = [&](int which) {
            const float(*v)[32] = part[which];
            return ((v[0][lane] + v[1][lane]) + (v[2][lane] + v[3][lane])) + ((v[4][lane] + v[5][lane]) + (v[6][lane] + v[7][lane]));
        };
        const float a = eight(0), b = eight(1);
        if (u < hidden) gW2[(size_t)t * hidden + u] = a;
        if (blockIdx.x == 0 && lane == 0) gb2[t] = b;
    }
}

// ---- gradients of the value encoding's projection and of the width weights, all layers ------------------------------------
//     gWpe[h][m][k] = sum_n gattn[n][h][m] psi[n][h][k],   gwpos[c] = sum_n galpha[n][c / 16] q[n][c]
// Block = (a share of the rows, layer); thread = (head, bin) with the head's sixteen channels in registers: psi is read
// once, coalesced, and bounds the kernel (2 KB per row and layer); gattn comes as shared-memory broadcasts.
constexpr int PE_ROWS = 16;  // rows staged at a time
constexpr int PE_PARTIAL = CH * 64 + CH;
constexpr int MAX_LAYERS = 32;
struct PeArgs {
    const float *gattn[MAX_LAYERS], *psi[MAX_LAYERS], *q[MAX_LAYERS], *galpha[MAX_LAYERS];
    float *gW[MAX_LAYERS], *gwpos[MAX_LAYERS];
    long long N;
    int shares;
    float *partial;
};

template <bool PSI>
__global__ void __launch_bounds__(512) pe_grad_kernel(const PeArgs p)
{
    __shared__ __align__(16) float go[PE_ROWS * CH];
    const int tid = threadIdx.x, l = blockIdx.y, h = tid >> 6;
    const long long lo = p.N * blockIdx.x / p.shares, hi = p.N * (blockIdx.x + 1) / p.shares;
    const float *gattn = p.gattn[l], *psi = PSI ? p.psi[l] : nullptr, *q = p.q[l], *galpha = p.galpha[l];
    float acc[16], wpos = 0.f, wpos_low = 0.f;
#pragma unroll
    for (int m = 0; m < 16; ++m) acc[m] = 0.f;
    for (long long n0 = lo; n0 < hi; n0 += PE_ROWS) {
        const int rows = (int)min((long long)PE_ROWS, hi - n0);
        if (PSI && psi != nullptr) {
            __syncthreads();
            for (int i = tid; i < rows * CH; i += 512) go[i] = gattn[n0 * CH + i];
            __syncthreads();
            float ps[PE_ROWS];
#pragma unroll
            for (int r = 0; r < PE_ROWS; ++r) ps[r] = r < rows ? psi[(n0 + r) * 512 + tid] : 0.f;
#pragma unroll
            for (int r = 0; r < PE_ROWS; ++r) {
                if (r >= rows) break;
                const float4 *g4 = reinterpret_cast<const float4 *>(go + r * CH + h * 16);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const float4 g = g4[m];
                    acc[4 * m] = fmaf(g.x, ps[r], acc[4 * m]); acc[4 * m + 1] = fmaf(g.y, ps[r], acc[4 * m + 1]);
                    acc[4 * m + 2] = fmaf(g.z, ps[r], acc[4 * m + 2]); acc[4 * m + 3] = fmaf(g.w, ps[r], acc[4 * m + 3]);
                }
            }
        }
        if (tid < CH && q != nullptr)
            for (int r = 0; r < rows; ++r)
                add_compensated(galpha[(n0 + r) * HEADS + (tid >> 4)] * (4.0f * q[(n0 + r) * CH + tid]), wpos, wpos_low);
    }
    float *out = p.partial + ((size_t)l * p.shares + blockIdx.x) * PE_PARTIAL;
    if (PSI) {
#pragma unroll
        for (int m = 0; m < 16; ++m) out[(h * 16 + m) * 64 + (tid & 63)] = acc[m];
    }
    if (tid < CH) out[CH * 64 + tid] = wpos + wpos_low;
}

// the shares added in a fixed order: block = 32 values, warp w the shares w, w + 8, ..., then the eight partial sums
__global__ void __launch_bounds__(256) pe_grad_sum_kernel(const PeArgs p, int first)
{
    __shared__ float part[8][32];
    const int l = blockIdx.y, lane = threadIdx.x & 31, w = threadIdx.x >> 5, idx = first + blockIdx.x * 32 + lane;
    const float *in = p.partial + (size_t)l * p.shares * PE_PARTIAL + idx;
    float t = 0.f;
#pragma unroll 4
    for (int sh = w; sh < p.shares; sh += 8) t += in[(size_t)sh * PE_PARTIAL];
    part[w][lane] = t;
    __syncthreads();
    if (w != 0) return;
    t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += part[i][lane];
    if (idx < CH * 64 && p.psi[l] == nullptr) return;  // (the layer's operators have written it, or it has none)
    if (idx < CH * 64) p.gW[l][idx] = t;
    else p.gwpos[l][idx - CH * 64] = t;
}

// ---- layers with a reciprocal-space half (domains "reci", "RECI", "multihead"): phi of either half, gradients of either ----
// phi = phi_real for heads below `real`, phi_reci for the others; the value encoding of the latter is zero
__global__ void merge_phi_kernel(const float4 *__restrict__ phi_real, const float4 *__restrict__ phi_reci, float4 *__restrict__ phi,
                                 float4 *__restrict__ values, long long E)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // (edge, half of the heads) x 16 float4
    const long long e = idx >> 4;
    const int t = (int)(idx & 15);
    if (e >= E) return;
    if (t < 2) phi[2 * e + t] = t == 0 ? phi_real[2 * e] : phi_reci[2 * e + 1];
    if (values != nullptr) values[32 * e + 16 + t] = make_float4(0.f, 0.f, 0.f, 0.f);
}
// the other way round: the gradient of phi split by heads, that of the reciprocal half's (zero) value encoding dropped
__global__ void split_gphi_kernel(const float4 *__restrict__ gphi, float4 *__restrict__ g_real, float4 *__restrict__ g_reci,
                                  float4 *__restrict__ gvalues, long long E)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long e = idx >> 4;
    const int t = (int)(idx & 15);
    if (e >= E) return;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < 2) {
        const float4 g = gphi[2 * e + t];
        g_real[2 * e + t] = t == 0 ? g : zero;
        g_reci[2 * e + t] = t == 0 ? zero : g;
    }
    if (gvalues != nullptr) gvalues[32 * e + 16 + t] = zero;
}
// ga of the halves side by side: heads 4-7 from the reciprocal sum
__global__ void merge_ga_kernel(const float4 *__restrict__ ga_reci, float4 *__restrict__ ga, long long N)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) ga[2 * i + 1] = ga_reci[2 * i + 1];
}

int projection_shares(long long rows)
{
    const long long most = (rows + PE_ROWS - 1) / PE_ROWS, cap = 2ll * sm_count();
    return (int)(most < 1 ? 1 : most < cap ? most : cap);
}

// ---- memory ----------------------------------------------------------------------------------------------------------------
enum Domain { REAL = 0, RECI = 1, RECI_INVERSE = 2, MULTIHEAD = 3 };
constexpr int SCALARS = 9;  // gauss_scale, gauss_shift, a_factor, elu_beta, lower_bound, dist_max, a_factor_hi, lower_bound_hi, domain
Domain domain_of(const cf_train_desc &d, int l) { return (Domain)(int)d.scalars[SCALARS * l + 8]; }
bool has_values(const cf_train_desc &d, int l) { return d.K > 0 && (domain_of(d, l) == REAL || domain_of(d, l) == MULTIHEAD); }

struct LayerSaved {
    unsigned char *forward, *backward;  // weight images
    float *q, *k, *v, *a, *attn, *psi, *y, *h;
    float *lse, *logit;                              // domain real: the fused attention
    unsigned char *left;                             // ... over pair grids: the rows left over, marked and listed
    int *leftover;
    float *phi_real, *sum_reci, *phi, *values, *prob;  // others: the operator pair
};
struct Saved {
    // memory whose size depends on atoms and crystals only
    int64_t *atom_start, *edge_start, *batch, *row_start;
    float *rvlen, *rvecs, *vcell;
    int32_t *row_order;
    unsigned *tickets;
    void *row_blocks;
    unsigned char *embed;
    float *x[MAX_LAYERS + 1];
    LayerSaved layer[MAX_LAYERS];
    float *pooled, *hid;
    size_t bytes;
    // memory whose size depends on the edges
    int64_t *edges;
    float *pos_ij, *kr, *phi_reci;
    void *lists, *grid;
    size_t edge_bytes;
};
Saved carve_saved(const cf_train_desc &d, void *memory, void *edge_memory, int64_t N, int64_t B, int64_t E)
{
    Carver c{static_cast<char *>(memory)};
    Saved s{};
    s.atom_start = c.take<int64_t>(B + 1);
    s.edge_start = c.take<int64_t>(B + 1);
    s.batch = c.take<int64_t>(N);
    s.row_start = c.take<int64_t>(N + 1);
    s.rvlen = c.take<float>(3 * B);
    s.rvecs = c.take<float>(9 * B);
    s.vcell = c.take<float>(B);
    s.row_order = c.take<int32_t>(N);
    s.tickets = c.take<unsigned>(MAX_LAYERS);
    s.row_blocks = c.take<unsigned>(row_blocks_words(N));
    s.embed = c.take<unsigned char>(TC_EMBED_BYTES);
    const size_t image = tc_image_bytes(tc_layer_blocks((int)d.ff_dim));
    for (int l = 0; l < d.num_layers; ++l) {
        LayerSaved &y = s.layer[l];
        s.x[l] = c.take<float>(N * CH);
        y.forward = c.take<unsigned char>(image);
        y.backward = c.take<unsigned char>(image);
        y.q = c.take<float>(N * CH); y.k = c.take<float>(N * CH); y.v = c.take<float>(N * CH);
        y.a = c.take<float>(N * HEADS); y.lse = c.take<float>(N * HEADS);
        y.attn = c.take<float>(N * CH);
        y.left = domain_of(d, l) == REAL ? c.take<unsigned char>(N) : nullptr;
        y.leftover = domain_of(d, l) == REAL ? c.take<int>(N) : nullptr;
        y.psi = d.K > 0 && domain_of(d, l) == REAL ? c.take<float>(N * HEADS * d.K) : nullptr;
        y.y = c.take<float>(N * CH);
        y.h = c.take<float>(N * d.ff_dim);
    }
    s.x[d.num_layers] = c.take<float>(N * CH);
    s.pooled = c.take<float>(B * CH);
    s.hid = c.take<float>(B * d.hidden);
    s.bytes = c.used;
    Carver e{static_cast<char *>(edge_memory)};
    s.edges = e.take<int64_t>(2 * E);
    s.pos_ij = e.take<float>(3 * E);
    bool fused = false, split = false;
    for (int l = 0; l < d.num_layers; ++l) {
        LayerSaved &y = s.layer[l];
        const Domain dom = domain_of(d, l);
        fused = fused || dom == REAL;
        split = split || dom != REAL;
        if (dom == REAL) {
            y.logit = e.take<float>(E * HEADS);
        } else {
            y.phi_real = dom == MULTIHEAD ? e.take<float>(E * HEADS) : nullptr;
            y.sum_reci = e.take<float>(E * HEADS);
            y.phi = e.take<float>(E * HEADS);
            y.values = has_values(d, l) ? e.take<float>(E * CH) : nullptr;
            y.prob = e.take<float>(E * HEADS);
        }
    }
    s.kr = split ? e.take<float>(3 * E) : nullptr;
    s.phi_reci = split ? e.take<float>(E * HEADS) : nullptr;
    const size_t lists = term_list_workspace_bytes(N, E), grid = pair_grid_reserve_training(N, B, E, d.K);
    s.lists = s.grid = fused ? e.take<char>(lists > grid ? lists : grid) : nullptr;  // (a step has one or the other)
    s.edge_bytes = e.used;
    return s;
}

struct LayerGrads {
    float *gh, *gy, *gattn, *gq, *gk, *gv, *ga;
};
struct Scratch {
    float *gx[MAX_LAYERS + 1];
    LayerGrads layer[MAX_LAYERS];
    float *glogit, *prob, *ghid, *partial, *pe_partial;
    float *gphi, *g_real, *g_reci, *gvalues, *ga_reci, *pair;  // the operator pair's backward
    int shares;
    size_t bytes;
};
int train_jobs(const cf_train_desc &d) { return d.num_layers * (4 + 2 * (int)(d.ff_dim / 128)) + 1 + (int)(d.hidden / 128); }
Scratch carve_scratch(const cf_train_desc &d, void *memory, int64_t N, int64_t B, int64_t E)
{
    Carver c{static_cast<char *>(memory)};
    Scratch s{};
    for (int l = 0; l < d.num_layers; ++l) {
        LayerGrads &g = s.layer[l];
        s.gx[l] = c.take<float>(N * CH);
        g.gh = c.take<float>(N * d.ff_dim);
        g.gy = c.take<float>(N * CH); g.gattn = c.take<float>(N * CH);
        g.gq = c.take<float>(N * CH); g.gk = c.take<float>(N * CH); g.gv = c.take<float>(N * CH);
        g.ga = c.take<float>(N * HEADS);
    }
    s.gx[d.num_layers] = c.take<float>(N * CH);
    s.glogit = c.take<float>(E * HEADS);
    s.prob = N >= PG_LEAST_ROWS ? c.take<float>(E * HEADS) : nullptr;
    bool split = false, values = false;
    for (int l = 0; l < d.num_layers; ++l) {
        split = split || domain_of(d, l) != REAL;
        values = values || (domain_of(d, l) != REAL && has_values(d, l));
    }
    if (split) {
        s.gphi = c.take<float>(E * HEADS); s.g_real = c.take<float>(E * HEADS); s.g_reci = c.take<float>(E * HEADS);
        s.ga_reci = c.take<float>(N * HEADS);
        s.gvalues = values ? c.take<float>(E * CH) : nullptr;
        s.pair = c.take<float>(values ? (size_t)cf_lattice_sum_bwd_proj_floats(E) : (size_t)E * HEADS);
    }
    s.ghid = c.take<float>(B * d.hidden);
    const int jobs = train_jobs(d);
    size_t most = 0;
    for (int at = 0; at < jobs; at += GRAD_MAX) {
        const size_t f = grad_partial_floats(jobs - at < GRAD_MAX ? jobs - at : GRAD_MAX, N);
        most = f > most ? f : most;
    }
    s.partial = c.take<float>(most);
    // shares of the rows per layer for the value-encoding gradient: one wave of blocks, at least one stage of rows each
    long long shares = sm_count() * 3 / (d.num_layers > 0 ? d.num_layers : 1);
    const long long most_shares = (N + PE_ROWS - 1) / PE_ROWS;
    shares = shares < most_shares ? shares : most_shares;
    s.shares = (int)(shares > 1 ? shares : 1);
    s.pe_partial = c.take<float>((size_t)d.num_layers * s.shares * PE_PARTIAL);
    s.bytes = c.used;
    return s;
}

int check_desc(const cf_train_desc *d, const char *who)
{
    CF_REQUIRE(d != nullptr && d->weights && d->scalars, CF_ERR_INVALID, "%s: null description", who);
    CF_REQUIRE(d->num_layers >= 1 && d->num_layers <= MAX_LAYERS, CF_ERR_UNSUPPORTED, "%s: %d layers (1..%d)", who, (int)d->num_layers, MAX_LAYERS);
    CF_REQUIRE(d->ff_dim > 0 && d->ff_dim % 128 == 0 && d->ff_dim <= TC_MAX_FF, CF_ERR_UNSUPPORTED,
               "%s: ff_dim=%lld must be a multiple of 128 up to %d", who, (long long)d->ff_dim, TC_MAX_FF);
    CF_REQUIRE(d->hidden > 0 && d->hidden % 128 == 0 && d->hidden <= 1024 && d->targets > 0, CF_ERR_UNSUPPORTED,
               "%s: head of %lld hidden units, %lld targets (a multiple of 128 up to 1024)", who, (long long)d->hidden, (long long)d->targets);
    CF_REQUIRE(d->feature_dim >= 1 && d->feature_dim <= 128, CF_ERR_UNSUPPORTED, "%s: %d features (1..128)", who, (int)d->feature_dim);
    CF_REQUIRE(d->K == 0 || d->K == 64, CF_ERR_UNSUPPORTED, "%s: K=%lld, only K in {0,64} is compiled", who, (long long)d->K);
    for (int l = 0; l < d->num_layers; ++l) {
        const double dom = d->scalars[SCALARS * l + 8];
        CF_REQUIRE(dom == REAL || ((dom == RECI || dom == RECI_INVERSE || dom == MULTIHEAD) && d->lattice_range <= 6), CF_ERR_UNSUPPORTED,
                   "%s: layer %d has domain code %g (0..3; lattice_range up to 6 for the reciprocal ones)", who, l, dom);
    }
    CF_REQUIRE(d->lattice_range >= 0 && d->lattice_range <= CF_MAX_RANGE && d->minimum_range >= 0, CF_ERR_RANGE,
               "%s: lattice_range %d outside [0,%d]", who, (int)d->lattice_range, CF_MAX_RANGE);
    return CF_OK;
}
enum Half { BEGIN, FORWARD, BACKWARD };
int check_batch(const cf_train_batch *b, const char *who, Half half)
{
    CF_REQUIRE(b != nullptr, CF_ERR_INVALID, "%s: null batch", who);
    CF_REQUIRE(b->N >= 1 && b->B >= 1 && b->B <= (1 << 20), CF_ERR_INVALID, "%s: empty batch or too many crystals", who);
    CF_REQUIRE(b->features && b->trans && b->saved && (half == BACKWARD || (b->pos && b->sizes)), CF_ERR_INVALID, "%s: null pointer", who);
    if (half == BEGIN) return CF_OK;
    CF_REQUIRE(b->E >= 1 && b->max_atoms >= 1 && b->max_atoms <= 1024, CF_ERR_RANGE, "%s: E=%lld, max_atoms=%lld (1..1024)", who,
               (long long)b->E, (long long)b->max_atoms);
    CF_REQUIRE(b->saved_edges, CF_ERR_INVALID, "%s: null pointer", who);
    return CF_OK;
}

// Weights of layer l: Wq Wk Wv b_in w_pos Wpe Wo bo W1 b1 W2 b2; after the layers: W_embed, the head's W1 b1 W2 b2.
enum { W_Q, W_K, W_V, B_IN, W_POS, W_PE, W_O, B_O, W_1, B_1, W_2, B_2, PER_LAYER };

bool lists_of(const cf_train_desc &d, const cf_train_batch &b, const Saved &s, TermList &list, float &a_widest)
{
    a_widest = -INFINITY;
    for (int l = 0; l < d.num_layers; ++l)
        if (domain_of(d, l) == REAL) a_widest = fmaxf(a_widest, (float)(d.scalars[SCALARS * l + 4] * d.scalars[SCALARS * l + 2]));
    const float floor = (float)b.floor_log2;
    if (s.lists == nullptr || !(floor > -200.0f) || !(a_widest < 0.0f)) return false;
    int *start, *count;
    float *dmin;
    unsigned long long *cursor;
    float2 *pool;
    term_list_carve(s.lists, b.N, b.E, &start, &count, &dmin, &cursor, &pool);
    list.pool = pool; list.start = start; list.count = count; list.dmin = dmin;
    list.window = term_window(floor, a_widest);
    return true;
}

// Whether a batch's layers of domain real go by pair grids, and what their calls share.  Both halves of a step decide alike, from the
// description, the sizes and the floor that the forward left in the batch (the process-wide one may change in between).  Nodes in
// reach are chosen for 2^-30, or for 2^-40 where terms are to be kept below 2^-30; a floor below that is not for nodes.
bool grid_of(const cf_train_desc &d, const cf_train_batch &b, const Saved &w, PairAttn &p, float &a_widest)
{
    a_widest = -INFINITY;
    double dist_max = 0.0;
    for (int l = 0; l < d.num_layers; ++l) {
        if (domain_of(d, l) != REAL) continue;
        const double dm = d.scalars[SCALARS * l + 5];
        if (d.K > 0 && dist_max != 0.0 && dm != dist_max) return false;  // (the nodes are those of one basis)
        dist_max = dm;
        a_widest = fmaxf(a_widest, (float)(d.scalars[SCALARS * l + 4] * d.scalars[SCALARS * l + 2]));
    }
    if (w.grid == nullptr || d.num_layers > PG_LAYERS || !pair_grid_pays_training(b.N, b.B, b.E, b.max_atoms, d.K)) return false;
    const float floor = (float)b.floor_log2;
    if (!(floor >= -40.0f) || !pair_grid_params(d.K, dist_max, d.wscale, a_widest, -30.0f, p.par)) return false;
    p.par.floor_log2 = floor < -30.0f ? -40.0f : -30.0f;
    p.rvlen = d.cutoff_radius != 0.0 ? w.rvlen : nullptr;
    p.atom_start = w.atom_start; p.edge_start = w.edge_start; p.N = b.N; p.B = b.B; p.E = b.E; p.K = d.K; p.max_atoms = (int)b.max_atoms;
    p.rule = BoxRule{(float)d.cutoff_radius, d.lattice_range, d.minimum_range};
    p.dist_max = dist_max; p.wscale = d.wscale;
    p.grid = pair_grid_carve(w.grid, b.N, b.B, b.E, d.K);
    return true;
}
// ... and one layer's
void grid_layer(PairAttn &p, const cf_train_desc &d, const LayerSaved &t, int l)
{
    p.q = t.q; p.k = t.k; p.v = t.v; p.a = t.a; p.W = d.weights[PER_LAYER * l + W_PE]; p.call = l; p.out = t.attn; p.lse = t.lse;
    p.psi_row = t.psi; p.logit = t.logit; p.left = t.left; p.leftover = t.leftover;
}

}  // namespace
}  // namespace cf

namespace cf {
// gW[h][m][k] = sum over rows of gv[row][h][m] psi[row][h][k] (the drop-in operator's projection gradient, rows = edges).
size_t projection_grad_floats(long long rows) { return (size_t)projection_shares(rows) * PE_PARTIAL; }
int launch_projection_grad(const float *gv, const float *psi, long long rows, float *gW, float *partial, cudaStream_t s)
{
    PeArgs pe{};
    pe.gattn[0] = gv; pe.psi[0] = psi; pe.gW[0] = gW;
    pe.N = rows; pe.shares = projection_shares(rows); pe.partial = partial;
    pe_grad_kernel<true><<<dim3(pe.shares, 1), 512, 0, s>>>(pe);
    pe_grad_sum_kernel<<<dim3(CH * 64 / 32, 1), 256, 0, s>>>(pe, 0);
    return launch_status("projection gradient");
}
}  // namespace cf

extern "C" int64_t cf_train_saved_bytes(const cf_train_desc *desc, int64_t N, int64_t B)
{
    if (cf::check_desc(desc, "cf_train_saved_bytes") != CF_OK) return -1;
    return (int64_t)cf::carve_saved(*desc, nullptr, nullptr, N, B, 0).bytes;
}

extern "C" int64_t cf_train_edge_bytes(const cf_train_desc *desc, int64_t N, int64_t B, int64_t E)
{
    if (cf::check_desc(desc, "cf_train_edge_bytes") != CF_OK) return -1;
    return (int64_t)cf::carve_saved(*desc, nullptr, nullptr, N, B, E).edge_bytes;
}

extern "C" int64_t cf_train_scratch_bytes(const cf_train_desc *desc, int64_t N, int64_t B, int64_t E)
{
    if (cf::check_desc(desc, "cf_train_scratch_bytes") != CF_OK) return -1;
    return (int64_t)cf::carve_scratch(*desc, nullptr, N, B, E).bytes;
}

namespace cf {
namespace {

// weight images of all layers, one direction (with the embedding's in the forward one)
int pack_all(const cf_train_desc &d, const Saved &w, bool forward, cudaStream_t s)
{
    static thread_local PackJob job;
    const int L = d.num_layers, ff = (int)d.ff_dim, blocks = tc_layer_blocks(ff);
    int count = 0, rc = CF_OK;
    if (forward) pack_embedding(job, count, w.embed, d.weights[PER_LAYER * L], d.feature_dim);
    for (int l = 0; l < L && rc == CF_OK; ++l) {
        const float *const *p = d.weights + PER_LAYER * l;
        if (count + blocks > PACK_MAX) {
            rc = launch_pack(job, count, s);
            count = 0;
        }
        (forward ? pack_layer_forward : pack_layer_backward)(job, count, forward ? w.layer[l].forward : w.layer[l].backward, ff, p[W_Q],
                                                             p[W_K], p[W_V], p[W_O], p[W_1], p[W_2]);
    }
    return rc == CF_OK ? launch_pack(job, count, s) : rc;
}

template <class Args>
void width_scalars(Args &t, const cf_train_desc &d, int l)
{
    const double *sc = d.scalars + SCALARS * l;
    t.gauss_scale = (float)sc[0]; t.gauss_shift = (float)sc[1]; t.a_factor = (float)sc[2];
    t.elu_beta = (float)sc[3]; t.lower_bound = (float)sc[4];
    t.a_factor_hi = (float)sc[6]; t.lower_bound_hi = (float)sc[7];
    t.inverse = domain_of(d, l) == RECI_INVERSE;
}

// the dense kernel before layer l's attention (l = num_layers: after the last one)
int forward_boundary(const cf_train_desc &d, const cf_train_batch &b, const Saved &w, int l, cudaStream_t s)
{
    DenseForward t{};
    t.N = b.N; t.ff = (int)d.ff_dim; t.chained = l > 0; t.weights_fresh = true;
    t.x_out = w.x[l];
    if (l > 0) {
        const LayerSaved &y = w.layer[l - 1];
        const float *const *p = d.weights + PER_LAYER * (l - 1);
        t.tail = y.forward; t.attn = y.attn; t.bo = p[B_O]; t.b1 = p[B_1]; t.b2 = p[B_2];
        t.x_in = w.x[l - 1]; t.y_save = y.y; t.h_save = y.h;
    } else {
        t.embed = w.embed; t.features = b.features; t.feature_dim = d.feature_dim;
    }
    if (l < d.num_layers) {
        const LayerSaved &y = w.layer[l];
        const float *const *p = d.weights + PER_LAYER * l;
        t.head = y.forward; t.bqkv = p[B_IN]; t.w_pos = p[W_POS];
        width_scalars(t, d, l);
        t.q = y.q; t.k = y.k; t.v = y.v; t.a = y.a;
    }
    return launch_dense_forward(t, s);
}

struct TrainBegin {
    const cf_train_desc *d;
    const cf_train_batch *b;
    const Saved *w;
};
int train_begin_launch(void *arg, cudaStream_t s)
{
    const TrainBegin &t = *static_cast<const TrainBegin *>(arg);
    const int rc = pack_all(*t.d, *t.w, true, s);
    return rc == CF_OK ? forward_boundary(*t.d, *t.b, *t.w, 0, s) : rc;
}

unsigned blocks_of(long long threads) { return (unsigned)((threads + 255) / 256); }

}  // namespace
}  // namespace cf

extern "C" int cf_train_begin(const cf_train_desc *desc, const cf_train_batch *batch, int64_t *counts, void **begun_event, void *stream)
{
    using namespace cf;
    int rc = check_desc(desc, "cf_train_begin");
    if (rc == CF_OK) rc = check_batch(batch, "cf_train_begin", BEGIN);
    if (rc != CF_OK) return rc;
    CF_REQUIRE(counts && begun_event, CF_ERR_INVALID, "cf_train_begin: null pointer");
    const Saved w = carve_saved(*desc, batch->saved, nullptr, batch->N, batch->B, 0);
    TrainBegin arg{desc, batch, &w};
    return read_sizes_beside(batch->sizes, batch->B, counts, as_stream(stream), train_begin_launch, &arg, begun_event);
}

extern "C" int cf_train_forward(const cf_train_desc *desc, cf_train_batch *batch, void *begun_event, float *y, void *stream)
{
    using namespace cf;
    int rc = check_desc(desc, "cf_train_forward");
    if (rc == CF_OK) rc = check_batch(batch, "cf_train_forward", FORWARD);
    if (rc != CF_OK) return rc;
    CF_REQUIRE(y && begun_event, CF_ERR_INVALID, "cf_train_forward: null pointer");
    batch->floor_log2 = weight_floor_log2();
    const cf_train_desc &d = *desc;
    const cf_train_batch &b = *batch;
    const int64_t N = b.N, B = b.B, E = b.E;
    const int L = d.num_layers;
    cudaStream_t s = as_stream(stream);
    const Saved w = carve_saved(d, b.saved, b.saved_edges, N, B, E);
    const float *const *tail_weights = d.weights + PER_LAYER * L;

    // ---- the backward's weight images behind the first dense block on the side stream (into memory that cf_train_begin has
    //      had), geometry and term lists here, beside both
    cudaStream_t side = early_prep_stream(nullptr, nullptr);
    CF_REQUIRE(side != nullptr, CF_ERR_CUDA, "cf_train_forward: the side stream could not be created");
    if (cudaMemsetAsync(w.tickets, 0, sizeof(unsigned) * MAX_LAYERS, s) != cudaSuccess) return launch_status("cf_train_forward: tickets");
    bool ordered = false;
    rc = launch_prepare_all(b.pos, b.trans, b.sizes, w.atom_start, w.edge_start, B, N, E, w.batch, w.edges, w.row_start, w.pos_ij, w.rvlen,
                            d.order_reach, w.row_order, &ordered, s, w.rvecs, w.vcell);
    if (rc != CF_OK) return rc;
    const int32_t *order = ordered ? w.row_order : nullptr;
    const float *rvlen = d.cutoff_radius != 0.0 ? w.rvlen : nullptr;
    TermList list{};
    PairAttn by_grid{};
    float a_widest;
    const bool gridded = grid_of(d, b, w, by_grid, a_widest);
    const bool listed = !gridded && lists_of(d, b, w, list, a_widest);
    if (gridded) {
        rc = launch_pair_grid_build(by_grid, w.pos_ij, b.trans, a_widest, nullptr, 0, 0, s);
        if (rc != CF_OK) return rc;
    }
    if (listed) {
        TermListBuild tb{};
        tb.pos_ij = w.pos_ij; tb.tvecs = b.trans; tb.rvlen = rvlen; tb.batch = w.batch; tb.edges = w.edges; tb.row_start = w.row_start;
        tb.row_order = order; tb.N = N; tb.E = E; tb.max_atoms = (int)b.max_atoms;
        tb.rule = BoxRule{(float)d.cutoff_radius, d.lattice_range, d.minimum_range};
        tb.a_widest = a_widest;
        tb.window = list.window;
        term_list_carve(w.lists, N, E, &tb.start, &tb.count, &tb.dmin, &tb.cursor, &tb.pool);
        tb.capacity = (long long)term_pool_entries(N, E);
        rc = launch_term_list_build(tb, s);
        if (rc != CF_OK) return rc;
    }
    static_assert(MAX_LAYERS <= ROW_BLOCK_LAYERS, "every layer has a scheduling block of its own");
    const RowBlocks row_blocks = row_blocks_carve(w.row_blocks, N);
    const bool by_blocks = listed && by_row_blocks(N, B, b.max_atoms);
    if (by_blocks) rc = launch_row_blocks(row_blocks, order, w.row_start, w.edges, N, E, s);
    if (rc != CF_OK) return rc;
    if (w.kr != nullptr) rc = cf_reci_phase(w.pos_ij, w.rvecs, w.batch, w.edges, E, w.kr, s);
    if (rc == CF_OK) rc = join_begun(begun_event, s);
    if (rc == CF_OK) rc = pack_all(d, w, false, side);  // (joined below)
    // ---- layers
    for (int l = 0; l < L && rc == CF_OK; ++l) {
        const LayerSaved &t = w.layer[l];
        const Domain dom = domain_of(d, l);
        const double dist_max = d.scalars[SCALARS * l + 5];
        if (dom == REAL && gridded) {
            grid_layer(by_grid, d, t, l);
            rc = grid_attn_impl(by_grid, w.pos_ij, b.trans, w.batch, w.edges, w.row_start, d.cutoff_radius, d.lattice_range, d.minimum_range, s);
        } else if (dom == REAL && by_blocks) {
            rc = block_attn_impl(t.q, t.k, t.v, t.a, w.pos_ij, b.trans, rvlen, w.batch, w.edges, w.row_start, N, B, E, d.K, b.max_atoms,
                                 dist_max, d.wscale, d.weights[PER_LAYER * l + W_PE], d.cutoff_radius, d.lattice_range, d.minimum_range,
                                 t.attn, t.logit, t.lse, t.psi, list, row_blocks, l, s);
        } else if (dom == REAL) {
            rc = infinite_attn_fwd_impl(t.q, t.k, t.v, t.a, nullptr, w.pos_ij, b.trans, rvlen, w.batch, w.edges, w.row_start, N, B, HEADS,
                                        HEAD_DIM, E, d.K, b.max_atoms, dist_max, d.wscale, d.weights[PER_LAYER * l + W_PE],
                                        d.cutoff_radius, d.lattice_range, d.minimum_range, t.attn, t.logit, t.lse, t.psi, order,
                                        listed ? &list : nullptr, w.tickets + l, s, true);
        } else {
            if (dom == MULTIHEAD)
                rc = cf_lattice_sum_fwd(t.a, 0, w.pos_ij, b.trans, w.batch, w.edges, N, HEADS, E, d.K, dist_max, d.wscale,
                                        d.weights[PER_LAYER * l + W_PE], 1, HEAD_DIM, rvlen, d.cutoff_radius, d.lattice_range,
                                        d.minimum_range, t.phi_real, t.values, s);
            float *phi_reci = dom == MULTIHEAD ? w.phi_reci : t.phi;
            if (rc == CF_OK)
                rc = cf_reci_sum_fwd(t.a, w.kr, w.rvecs, w.vcell, w.batch, w.row_start, N, HEADS, E, d.lattice_range, phi_reci, t.sum_reci, s);
            if (dom == MULTIHEAD && rc == CF_OK)
                merge_phi_kernel<<<blocks_of(16 * E), 256, 0, s>>>(reinterpret_cast<const float4 *>(t.phi_real),
                                                                   reinterpret_cast<const float4 *>(phi_reci),
                                                                   reinterpret_cast<float4 *>(t.phi), reinterpret_cast<float4 *>(t.values), E);
            if (rc == CF_OK) rc = cf_fused_attn_fwd(t.q, t.k, t.v, t.phi, t.values, w.edges, w.row_start, N, HEADS, HEAD_DIM, E, t.prob, t.attn, s);
        }
        if (rc == CF_OK) rc = forward_boundary(d, b, w, l + 1, s);
    }
    if (rc == CF_OK)
        rc = launch_pool_head(w.x[L], w.atom_start, tail_weights[1], tail_weights[2], tail_weights[3], tail_weights[4], (int)d.hidden,
                              (int)d.targets, B, y, w.pooled, w.hid, true, s);
    const int joined = join_early_prep(s);  // (after an error too: the images may still be being written)
    return rc == CF_OK ? joined : rc;
}

extern "C" int cf_train_backward(const cf_train_desc *desc, const cf_train_batch *batch, const float *gy, void *scratch,
                                 float *const *grads, void *stream)
{
    using namespace cf;
    int rc = check_desc(desc, "cf_train_backward");
    if (rc == CF_OK) rc = check_batch(batch, "cf_train_backward", BACKWARD);
    if (rc != CF_OK) return rc;
    CF_REQUIRE(gy && scratch && grads, CF_ERR_INVALID, "cf_train_backward: null pointer");
    const cf_train_desc &d = *desc;
    const cf_train_batch &b = *batch;
    const int64_t N = b.N, B = b.B, E = b.E;
    const int L = d.num_layers, ff = (int)d.ff_dim, hidden = (int)d.hidden, targets = (int)d.targets;
    cudaStream_t s = as_stream(stream);
    const Saved w = carve_saved(d, b.saved, b.saved_edges, N, B, E);
    Scratch g = carve_scratch(d, scratch, N, B, E);
    const float *const *tail_weights = d.weights + PER_LAYER * L;
    float *const *tail_grads = grads + PER_LAYER * L;
    const int32_t *order = rows_are_ordered(B, N) ? w.row_order : nullptr;
    const float *rvlen = d.cutoff_radius != 0.0 ? w.rvlen : nullptr;
    TermList list{};
    PairAttn by_grid{};
    float a_widest;
    const bool gridded = grid_of(d, b, w, by_grid, a_widest);
    const bool listed = !gridded && lists_of(d, b, w, list, a_widest);

    head_backward_kernel<<<(unsigned)B, 128, 0, s>>>(gy, w.hid, tail_weights[1], tail_weights[3], w.atom_start, hidden, targets, g.ghid, g.gx[L]);
    head_weight_grad_kernel<<<dim3((hidden + 31) / 32, targets), 256, 0, s>>>(gy, w.hid, B, hidden, targets, tail_grads[3], tail_grads[4]);
    for (int l = L - 1; l >= -1 && rc == CF_OK; --l) {
        DenseBackward t{};
        t.N = N; t.ff = ff;
        t.gx = g.gx[l + 1];
        if (l + 1 < L) {  // head of layer l + 1
            const LayerSaved &y = w.layer[l + 1];
            const LayerGrads &gg = g.layer[l + 1];
            t.head = y.backward; t.q = y.q; t.w_pos = d.weights[PER_LAYER * (l + 1) + W_POS];
            width_scalars(t, d, l + 1);
            t.gq = gg.gq; t.gk = gg.gk; t.gv = gg.gv; t.ga = gg.ga; t.g_res = gg.gy;
        }
        if (l >= 0) {
            const LayerSaved &y = w.layer[l];
            const LayerGrads &gg = g.layer[l];
            t.tail = y.backward; t.h = y.h; t.gh = gg.gh; t.gy = gg.gy; t.gattn = gg.gattn;
        }
        rc = launch_dense_backward(t, s);
        if (rc != CF_OK || l < 0) break;
        const LayerSaved &y = w.layer[l];
        const LayerGrads &gg = g.layer[l];
        const double dist_max = d.scalars[SCALARS * l + 5];
        if (domain_of(d, l) == REAL && gridded) {
            grid_layer(by_grid, d, y, l);
            by_grid.gout = gg.gattn; by_grid.gq = gg.gq; by_grid.gk = gg.gk; by_grid.gv = gg.gv; by_grid.ga = gg.ga;
            by_grid.glogit = g.glogit; by_grid.prob = g.prob;
            rc = grid_attn_bwd_impl(by_grid, w.pos_ij, b.trans, w.batch, w.edges, w.row_start, s);
            continue;
        }
        if (domain_of(d, l) == REAL) {
            rc = infinite_attn_bwd_impl(y.q, y.k, y.v, y.a, nullptr, w.pos_ij, b.trans, rvlen, w.batch, w.edges, w.row_start, N, B, HEADS,
                                        HEAD_DIM, E, d.K, b.max_atoms, dist_max, d.wscale, d.weights[PER_LAYER * l + W_PE],
                                        d.cutoff_radius, d.lattice_range, d.minimum_range, y.logit, y.lse, y.attn, gg.gattn, gg.gq, gg.gk,
                                        gg.gv, gg.ga, g.glogit, order, listed ? &list : nullptr, s);
            continue;
        }
        const bool multi = domain_of(d, l) == MULTIHEAD;
        rc = cf_fused_attn_bwd(y.q, y.k, y.v, y.values, w.edges, w.row_start, N, HEADS, HEAD_DIM, E, y.prob, y.attn, gg.gattn, gg.gq, gg.gk,
                               gg.gv, g.gphi, y.values != nullptr ? g.gvalues : nullptr, s);
        if (multi && rc == CF_OK) {
            split_gphi_kernel<<<blocks_of(16 * E), 256, 0, s>>>(reinterpret_cast<const float4 *>(g.gphi), reinterpret_cast<float4 *>(g.g_real),
                                                                reinterpret_cast<float4 *>(g.g_reci),
                                                                reinterpret_cast<float4 *>(y.values != nullptr ? g.gvalues : nullptr), E);
            if (y.values != nullptr)
                rc = cf_lattice_sum_bwd_proj(y.a, w.pos_ij, b.trans, w.batch, w.edges, w.row_start, y.phi_real, g.g_real, g.gvalues,
                                             d.weights[PER_LAYER * l + W_PE], N, HEADS, E, d.K, dist_max, d.wscale, rvlen, d.cutoff_radius,
                                             d.lattice_range, d.minimum_range, gg.ga, grads[PER_LAYER * l + W_PE], g.pair, s);
            else
                rc = cf_lattice_sum_bwd(y.a, w.pos_ij, b.trans, w.batch, w.edges, w.row_start, y.phi_real, g.g_real, nullptr, N, HEADS, E, 0,
                                        dist_max, d.wscale, rvlen, d.cutoff_radius, d.lattice_range, d.minimum_range, gg.ga, nullptr, g.pair, s);
        }
        if (rc == CF_OK)
            rc = cf_reci_sum_bwd(y.a, w.kr, w.rvecs, w.batch, w.row_start, multi ? g.g_reci : g.gphi, y.sum_reci, N, HEADS, E, d.lattice_range,
                                 multi ? g.ga_reci : gg.ga, s);
        if (multi && rc == CF_OK)
            merge_ga_kernel<<<blocks_of(N), 256, 0, s>>>(reinterpret_cast<const float4 *>(g.ga_reci), reinterpret_cast<float4 *>(gg.ga), N);
    }
    if (rc != CF_OK) return rc;
    // ---- value encoding and width weights
    PeArgs pe{};
    pe.N = N; pe.shares = g.shares; pe.partial = g.pe_partial;
    for (int l = 0; l < L; ++l) {
        pe.gattn[l] = g.layer[l].gattn; pe.psi[l] = w.layer[l].psi; pe.q[l] = w.layer[l].q; pe.galpha[l] = g.layer[l].ga;
        pe.gW[l] = grads[PER_LAYER * l + W_PE]; pe.gwpos[l] = grads[PER_LAYER * l + W_POS];
    }
    if (d.K > 0) pe_grad_kernel<true><<<dim3(g.shares, L), 512, 0, s>>>(pe);
    else pe_grad_kernel<false><<<dim3(g.shares, L), 512, 0, s>>>(pe);
    pe_grad_sum_kernel<<<dim3((d.K > 0 ? PE_PARTIAL : CH) / 32, L), 256, 0, s>>>(pe, d.K > 0 ? 0 : CH * 64);
    // ---- projections
    static thread_local GradJobs jobs;
    int count = 0;
    auto add = [&](const float *gm, int ldg, const float *xm, int ldx, long long rows, int x_cols, float *out, int ldo, float *bias) {
        if (rc == CF_OK && count == GRAD_MAX) {
            rc = launch_weight_grads(jobs, count, g.partial, s);
            count = 0;
        }
        GradJob &j = jobs.j[count++];
        j.g = gm; j.ldg = ldg; j.x = xm; j.ldx = ldx; j.rows = rows; j.x_cols = x_cols; j.out = out; j.ldo = ldo; j.bias = bias;
    };
    for (int l = 0; l < L; ++l) {
        const LayerSaved &y = w.layer[l];
        const LayerGrads &gg = g.layer[l];
        float *const *o = grads + PER_LAYER * l;
        add(gg.gq, CH, w.x[l], CH, N, CH, o[W_Q], CH, o[B_IN]);
        add(gg.gk, CH, w.x[l], CH, N, CH, o[W_K], CH, o[B_IN] + CH);
        add(gg.gv, CH, w.x[l], CH, N, CH, o[W_V], CH, o[B_IN] + 2 * CH);
        add(gg.gy, CH, y.attn, CH, N, CH, o[W_O], CH, o[B_O]);
        for (int c = 0; c < ff / CH; ++c) {
            add(gg.gh + c * CH, ff, y.y, CH, N, CH, o[W_1] + (size_t)c * CH * CH, CH, o[B_1] + c * CH);
            add(g.gx[l + 1], CH, y.h + c * CH, ff, N, CH, o[W_2] + c * CH, ff, c == 0 ? o[B_2] : nullptr);
        }
    }
    add(g.gx[0], CH, b.features, (int)d.feature_dim, N, (int)d.feature_dim, tail_grads[0], (int)d.feature_dim, nullptr);
    for (int u = 0; u < hidden / CH; ++u)
        add(g.ghid + u * CH, hidden, w.pooled, CH, B, CH, tail_grads[1] + (size_t)u * CH * CH, CH, tail_grads[2] + u * CH);
    if (rc == CF_OK) rc = launch_weight_grads(jobs, count, g.partial, s);
    if (rc != CF_OK) return rc;
    return launch_status("cf_train_backward");
}
