// Pair grids (pair_grid.cuh): the plan of a batch and the vectors of its pairs.
#include "pair_grid.cuh"

#include "lattice_core.cuh"
#include "mma_frag.cuh"

namespace cf {
namespace {

// ---- plan: boxes, units and row tiles of a batch; fragments of the basis ---------------------------------------------------
constexpr int PLAN_THREADS = 1024;
constexpr int TILE_CLASSES = PG_MAX_ATOMS / PG_ROWS + 1;

struct PlanArgs {
    const int64_t *atom_start, *edge_start;
    const float *rvlen;
    long long N, B, E, tile_cap, extra_cap;
    BoxRule rule;
    float a_widest;
    double wscale;
    int basis_blocks, calls;     // blocks of the two kinds
    float wscale_f, bits;        // g_k(d_m) = 2^(bits u^2), u = (m - 5) wscale - 3 (k + 1)
    const float *W[PG_LAYERS];
    PairGrid grid;
};

// The value projection of one (call, head) at the nodes, V[m] = sum_k W[:, k] g_k(d_m): 16 channels x 16 nodes per fragment, in half
// pairs scaled to a largest value between 2^13 and 2^14.  Warp = node tile.
__device__ __forceinline__ void projected_basis(const PlanArgs &p, int at, float *w, unsigned *largest)
{
    constexpr int LD = 65;
    const int tid = threadIdx.x, lane = tid & 31, mt = tid >> 5, h = at % HEADS;
    if (tid == 0) *largest = 0u;
    for (int i = tid; i < HEAD_DIM * 64; i += blockDim.x) w[(i >> 6) * LD + (i & 63)] = p.W[at / HEADS][h * HEAD_DIM * 64 + i];
    __syncthreads();
    const int g = lane >> 2, t = lane & 3;
    float v[4][2];  // channels g, g + 8; nodes 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u][0] = v[u][1] = 0.f;
    if (mt < PG_TILES_BASIS) {
        for (int k = 0; k < 64; ++k) {
            const float w0 = w[g * LD + k], w1 = w[(g + 8) * LD + k];
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const float u = (float)(mt * PG_TILE + 2 * t + 8 * c + x - PG_BELOW) * p.wscale_f - 3.0f * (float)(k + 1);  // (whole numbers where wscale = 1)
                    const float b = exp2f(p.bits * (u * u));
                    v[2 * c][x] = fmaf(w0, b, v[2 * c][x]);
                    v[2 * c + 1][x] = fmaf(w1, b, v[2 * c + 1][x]);
                }
        }
        float most = 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) most = fmaxf(most, fmaxf(fabsf(v[u][0]), fabsf(v[u][1])));
        atomicMax(largest, __float_as_uint(most));
    }
    __syncthreads();
    const unsigned x = min(max(*largest & 0x7f800000u, 30u << 23), 230u << 23);
    if (mt < PG_TILES_BASIS) {
        const float scale = __uint_as_float((267u << 23) - x);
        unsigned hi[4], lo[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) split_f16(v[u][0] * scale, v[u][1] * scale, hi[u], lo[u]);
        uint4 *out = p.grid.projected + ((size_t)at * PG_TILES_BASIS + mt) * 64 + lane;
        out[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        out[32] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
    if (tid == 0) p.grid.projected_scale[at] = __uint_as_float(x - (13u << 23));
}

// ... by itself, for batches that are prepared ahead of the weights' stream
__global__ void __launch_bounds__(32 * PG_TILES_BASIS) projected_basis_kernel(const PlanArgs p)
{
    __shared__ float w_sh[HEAD_DIM * 65];
    __shared__ unsigned largest;
    projected_basis(p, blockIdx.x, w_sh, &largest);
}

__device__ __forceinline__ float basis_at_node(int m, int k, double wscale)
{
    const double u = ((double)(m - PG_BELOW) * wscale - 3.0 * (double)(k + 1)) / (3.0 * wscale);  // in standard deviations
    return (float)exp2(-0.72134752044448170 * u * u) * PG_BASIS_SCALE;
}

__device__ __forceinline__ long long block_scan(long long v, long long *warp_totals, long long &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += u;
    }
    __syncthreads();
    if (lane == 31) warp_totals[w] = x;
    __syncthreads();
    long long before = 0, all = 0;
#pragma unroll 4
    for (int i = 0; i < PLAN_THREADS / 32; ++i) {
        const long long t = warp_totals[i];
        before += i < w ? t : 0;
        all += t;
    }
    total = all;
    return before + x - v;
}

// Block 0: one thread per crystal.  The tiles are listed by size, largest crystals first, so that the last blocks of an
// attention launch are short ones.  The other blocks: the basis fragments, a thread per (fragment, lane); the projected basis, a
// block per (call, head).
__global__ void __launch_bounds__(PLAN_THREADS) pair_plan_kernel(const PlanArgs p)
{
    const int tid = threadIdx.x;
    __shared__ float w_sh[HEAD_DIM * 65];
    __shared__ unsigned largest;
    if ((int)blockIdx.x > p.basis_blocks) {
        projected_basis(p, blockIdx.x - 1 - p.basis_blocks, w_sh, &largest);
        return;
    }
    if (blockIdx.x > 0) {
        const int at = (blockIdx.x - 1) * PLAN_THREADS + tid, frag = (at >> 5) % PG_FRAGS, lane = at & 31;
        const bool nodes = (at >> 5) >= PG_FRAGS;
        if ((at >> 5) >= 2 * PG_FRAGS) return;
        const int mt = frag >> 2, bt = frag & 3, g = lane >> 2, t = lane & 3;
        unsigned hi[4], lo[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = g + 8 * (u & 1), c = 2 * t + 8 * (u >> 1);
            float v[2];
#pragma unroll
            for (int x = 0; x < 2; ++x)
                v[x] = nodes ? basis_at_node(mt * 16 + r, bt * 16 + c + x, p.wscale) : basis_at_node(mt * 16 + c + x, bt * 16 + r, p.wscale);
            split_f16(v[0], v[1], hi[u], lo[u]);
        }
        uint4 *out = (nodes ? p.grid.basis_nodes : p.grid.basis) + (size_t)frag * 64 + lane;
        out[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        out[32] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        return;
    }
    __shared__ long long totals[PLAN_THREADS / 32];
    __shared__ int hist[TILE_CLASSES + 1], cursor[TILE_CLASSES + 1];
    for (int i = tid; i < 4 * (PG_LAYERS + 1); i += PLAN_THREADS) p.grid.counters[i] = 0u;
    for (int i = tid; i <= TILE_CLASSES; i += PLAN_THREADS) hist[i] = 0;
    __syncthreads();
    const long long pairs_all = (p.E + p.N) / 2;
    long long extra_before = 0, units_before = 0;
    for (long long c0 = 0; c0 < p.B; c0 += PLAN_THREADS) {
        const long long c = c0 + tid;
        long long n = 0, pairs = 0;
        int rmin = 0, e1 = 1, e2 = 1, e3 = 1;
        bool fits = false, all = false;
        if (c < p.B) {
            n = p.atom_start[c + 1] - p.atom_start[c];
            pairs = n * (n + 1) / 2;
            fits = n > 0 && n <= PG_MAX_ATOMS && (p.edge_start[c] + p.atom_start[c]) / 2 + pairs <= pairs_all;
            const float *rv = p.rvlen != nullptr ? p.rvlen + 3 * c : nullptr;
            rmin = packed_box(p.rule, -INFINITY, rv);
            const int rmax = packed_box(p.rule, p.a_widest, rv);
            e1 = box_r1(rmax) - box_r1(rmin) + 1; e2 = box_r2(rmax) - box_r2(rmin) + 1; e3 = box_r3(rmax) - box_r3(rmin) + 1;
            all = e1 >= 1 && e2 >= 1 && e3 >= 1 && (long long)e1 * e2 * e3 <= PG_MAX_VARIANTS;
            if (!all) e1 = e2 = e3 = 1;  // (only the smallest box)
        }
        long long total;
        const long long want = fits ? ((long long)e1 * e2 * e3 - 1) * pairs : 0;
        const long long at = extra_before + block_scan(want, totals, total);
        extra_before += total;
        if (at + want > p.extra_cap) {
            e1 = e2 = e3 = 1;
            all = false;
        }
        const long long units = fits ? (long long)e1 * e2 * e3 * ((pairs + PG_UNIT - 1) / PG_UNIT) : 0;
        const long long unit = units_before + block_scan(units, totals, total);
        units_before += total;
        if (c < p.B) {
            p.grid.info[c] = make_int4(rmin, e1 | (e2 << 8) | (e3 << 16) | (all ? PG_ALL_BOXES : 0), (int)(pairs_all + at), fits ? (int)n : -1);
            p.grid.unit_start[c] = (int)unit;
            if (n > 0) atomicAdd(&hist[min((int)((n + PG_ROWS - 1) / PG_ROWS), TILE_CLASSES)], (int)((n + PG_ROWS - 1) / PG_ROWS));
        }
    }
    __syncthreads();
    if (tid == 0) {
        p.grid.unit_start[p.B] = (int)units_before;
        int at = 0;
        for (int i = TILE_CLASSES; i >= 0; --i) { cursor[i] = at; at += hist[i]; }
        p.grid.counters[0] = (unsigned)min((long long)at, p.tile_cap);
    }
    __syncthreads();
    for (long long c = tid; c < p.B; c += PLAN_THREADS) {
        const int n = (int)(p.atom_start[c + 1] - p.atom_start[c]), count = (n + PG_ROWS - 1) / PG_ROWS;
        if (count <= 0) continue;
        const int at = atomicAdd(&cursor[min(count, TILE_CLASSES)], count);
        const int4 info = p.grid.info[c];  // (this thread's own)
        const int a0 = (int)p.atom_start[c], first = (int)((p.edge_start[c] + a0) / 2);
        for (int i = 0; i < count && at + i < p.tile_cap; ++i) {
            p.grid.tiles[2 * (at + i)] = make_int4((int)c, i * PG_ROWS, info.w == n ? n : -n, a0);
            p.grid.tiles[2 * (at + i) + 1] = make_int4(first, info.z, info.x, info.y);
        }
    }
}

// ---- vectors ----------------------------------------------------------------------------------------------------------------
// Interpolation weights of node floor(x) - 5 + q, y = x - floor(x) - 1/2: sum_p COEF[q][p] y^p; those of q and 11 - q mirror each
// other.  Least squares (degree nine, 1e-10) to the kriging weights C^-1 c(y), C_ab = exp(-(a - b)^2 / 4 s^2), c_a = exp(-(a -
// x)^2 / 4 s^2): the autocorrelation of a Gaussian of s node spacings, a, b the twelve nodes.  s = 3 with a basis; without one s =
// 6, since far out a Gaussian of sigma is exp(-d y / sigma^2) from node to node and its value there counts relative to
// itself (keys with large logits): 2e-8 at four sigma, where s = 3 leaves 1e-5.
struct Coefs {
    float k[6][10];
};
__device__ constexpr Coefs COEF_PLAIN = {{
    {-0.000147784926f, 2.68830511e-05f, 0.000700840342f, -0.000127487888f, -0.000462355314f, 8.41072638e-05f, 9.60860564e-05f, -1.74786376e-05f, -7.50003651e-06f, 1.36208806e-06f},
    {0.00185552736f, -0.000412473627f, -0.00876917505f, 0.0019493463f, 0.00566300064f, -0.0012588827f, -0.00111877848f, 0.000248703388f, 7.93026382e-05f, -1.76053873e-05f},
    {-0.0112932083f, 0.00322726628f, 0.053007211f, -0.0151479505f, -0.0327750117f, 0.0093663624f, 0.00583629827f, -0.00166791739f, -0.00034519365f, 9.85384863e-05f},
    {0.0455242983f, -0.0182115487f, -0.210110911f, 0.0840530981f, 0.115945637f, -0.0463842237f, -0.0157627848f, 0.00630626871f, 0.000798926085f, -0.000319303168f},
    {-0.147652146f, 0.098438324f, 0.639468618f, -0.426329408f, -0.200881522f, 0.133932628f, 0.0220170595f, -0.014680277f, -0.00100614225f, 0.000670223851f},
    {0.611713313f, -1.22343154f, -0.474296583f, 0.948616636f, 0.112510251f, -0.225036538f, -0.0110678805f, 0.0221388439f, 0.000480607212f, -0.000960459596f},
}};
__device__ constexpr Coefs COEF_BASIS = {{
    {-0.000264721665f, 4.85051069e-05f, 0.0012604898f, -0.000230972713f, -0.000852433915f, 0.000156250544f, 0.000188266416f, -3.45318413e-05f, -1.67243168e-05f, 3.06495886e-06f},
    {0.0027411572f, -0.000612315369f, -0.0130074548f, 0.00290574171f, 0.00861599781f, -0.00192536726f, -0.00181601493f, 0.000406109797f, 0.000148963987f, -3.32983128e-05f},
    {-0.0142998786f, 0.00409854429f, 0.0673952253f, -0.0193174616f, -0.0427967533f, 0.0122710769f, 0.00820092407f, -0.00235345447f, -0.000581145217f, 0.000166796133f},
    {0.0513506738f, -0.0205732775f, -0.237991165f, 0.0953547303f, 0.135360771f, -0.0542557395f, -0.0203414117f, 0.00816303065f, 0.00125536198f, -0.000503997355f},
    {-0.154194412f, 0.102855756f, 0.670773729f, -0.447467683f, -0.222678338f, 0.148653016f, 0.0271555793f, -0.0181513495f, -0.00151806504f, 0.00101527029f},
    {0.614667174f, -1.22941339f, -0.488430788f, 0.977240576f, 0.12235073f, -0.244968284f, -0.013387337f, 0.0268379255f, 0.000711607978f, -0.00142742543f},
}};

constexpr int UNIT = PG_UNIT;                   // pairs of a warp, four lanes each
constexpr int LIST = 24;                        // places of a lane waiting for their nodes
constexpr int AT_ONCE = 2;                      // places that a lane works on at a time
constexpr int ROOM = 5;                         // images between two looks at the lists: the usual box's column
constexpr int BUILD_WARPS = 4, BUILD_BLOCKS = 5;
constexpr int MAX_RUN = 4;                      // units in a row that a warp takes
__host__ __device__ constexpr size_t build_smem(int tiles) { return BUILD_WARPS * sizeof(float) * ((size_t)(tiles * PG_TILE + PG_POINTS) * UNIT + LIST * 32); }

struct BuildArgs {
    const float *pos_ij, *tvecs;
    const int64_t *atom_start, *edge_start;
    long long B;
    float inv_h2, inv_h2_low;
    PairGrid grid;
};

// The last crystal whose first unit is not beyond u: a 32-way search by the whole warp.
__device__ __forceinline__ int crystal_of_unit(const int *unit_start, int B, int u, int lane)
{
    int lo = 0, len = B;  // the answer lies in [lo, lo + len)
    while (len > 1) {
        const int step = (len + 31) / 32, at = lo + lane * step;
        const unsigned m = __ballot_sync(FULL, lane * step < len && unit_start[at] <= u);
        const int k = 31 - __clz(m);  // (bit 0 is always set)
        len = min(step, len - k * step);
        lo += k * step;
    }
    return lo;
}

// One warp per eight pairs, lane = (quarter, pair).  The four lanes of a pair deal the columns of the box among themselves and
// list the images in range; then all four walk the four lists, each with three of the twelve nodes of an image's place x = d / h:
// the nodes of one place are disjoint, places come one after the other, so there are no conflicts and no atomics, and a pair's
// images add in a fixed order.  In shared memory node m of pair p lies in bank 8 m + p: a quarter's nodes are 3 apart from the next
// one's, so the 32 lanes meet no bank twice.
// Bound by instruction issue and the waits of a lane's chain (0.73 M vectors of 1,024 crystals of up to 60 atoms: 410 us; their
// bytes 80).  So two places are worked on at a time, without spills (95 registers, twenty warps on an SM; at 80 and twenty-four
// 465 us, three or four places at 114 and sixteen 415 and 425), and since a unit's images differ by a factor of ten, warps take
// units as they come free: 256 crystals of up to 40 atoms 80 us, 190 with equal shares and one place at a time; 128 of up to 30 30
// and 36 us.  One pair per lane, with all twelve nodes in its own column, left room for seven warps: 591 us and 63.
template <int TILES>
__global__ void __launch_bounds__(32 * BUILD_WARPS, BUILD_BLOCKS) pair_grid_kernel(const BuildArgs p)
{
    extern __shared__ __align__(16) float build_mem[];
    const int lane = threadIdx.x & 31, quarter = lane >> 3, mine = lane & 7;
    // [node][pair], and as many nodes as a place has that nobody reads; [LIST][32]
    float *hist = build_mem + (threadIdx.x >> 5) * ((TILES * PG_TILE + PG_POINTS) * UNIT + LIST * 32);
    unsigned *list = reinterpret_cast<unsigned *>(hist + (TILES * PG_TILE + PG_POINTS) * UNIT);
    constexpr int NODES = TILES * PG_TILE;
    constexpr Coefs COEF = TILES == PG_TILES_BASIS ? COEF_BASIS : COEF_PLAIN;
    // the quarter's nodes 3 quarter ... + 2: of either half of the twelve the upper one mirrors the lower
    float2 k[3][5];
#pragma unroll
    for (int n = 0; n < 3; ++n)
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            const float e0 = COEF.k[n][2 * d], o0 = COEF.k[n][2 * d + 1], e1 = COEF.k[3 + n][2 * d], o1 = COEF.k[3 + n][2 * d + 1];
            const float e2 = COEF.k[5 - n][2 * d], o2 = -COEF.k[5 - n][2 * d + 1], e3 = COEF.k[2 - n][2 * d], o3 = -COEF.k[2 - n][2 * d + 1];
            k[n][d] = make_float2(PG_RHO_SCALE * (quarter < 2 ? (quarter == 0 ? e0 : e1) : (quarter == 2 ? e2 : e3)),
                                  PG_RHO_SCALE * (quarter < 2 ? (quarter == 0 ? o0 : o1) : (quarter == 2 ? o2 : o3)));
        }
    const int units = p.grid.unit_start[p.B], warps = gridDim.x * BUILD_WARPS;
    const int length = max(1, min(MAX_RUN, units / (4 * warps)));
    int c = 0, c_begin = 0, c_end = 0;  // the crystal and its units
    int4 info = make_int4(0, 0, 0, 0);
    Cell cell;
    float inv_t3sq = 0.f;
    // runs of units: the first by the warp's number, the others as warps come free (a unit's images differ by a factor of ten)
    int run = (blockIdx.x * BUILD_WARPS + (threadIdx.x >> 5)) * length, u = run, ticket = 0;
    auto next_unit = [&]() {
        if (++u < run + length) return;
        u = run = warps * length + __shfl_sync(FULL, ticket, 0);
    };
    for (; u < units; next_unit()) {
        if (u == run && lane == 0) ticket = (int)atomicAdd(p.grid.counters + 1, (unsigned)length);
        if (u < c_begin || u >= c_end) {
            c = crystal_of_unit(p.grid.unit_start, (int)p.B, u, lane);
            c_begin = p.grid.unit_start[c];
            c_end = p.grid.unit_start[c + 1];
            info = p.grid.info[c];
            cell.load(p.tvecs + 9 * (long long)c);
            inv_t3sq = __frcp_rn(fmaf(cell.t3z, cell.t3z, fmaf(cell.t3y, cell.t3y, cell.t3x * cell.t3x)));
        }
        const int n = info.w, pairs = n * (n + 1) / 2, per_variant = (pairs + UNIT - 1) / UNIT;
        int local = u - c_begin, variant = 0;
        int R1 = box_r1(info.x), R2 = box_r2(info.x), R3 = box_r3(info.x);
        if (local >= per_variant) {
            variant = local / per_variant;
            local -= variant * per_variant;
            const int e1 = info.y & 0xff, e2 = (info.y >> 8) & 0xff;
            R1 += variant % e1; R2 += variant / e1 % e2; R3 += variant / (e1 * e2);
        }
        const int first = local * UNIT, pair = min(first + mine, pairs - 1);
        // row and column of the pair: rows i start at i n - i (i - 1) / 2
        int i = (int)(0.5f * ((float)(2 * n + 1) - sqrtf((float)((2 * n + 1) * (2 * n + 1) - 8 * pair))));
        i = max(0, min(i, n - 1));
        while (i > 0 && i * n - i * (i - 1) / 2 > pair) --i;
        while (i + 1 < n && (i + 1) * n - (i + 1) * i / 2 <= pair) ++i;
        const int j = i + pair - (i * n - i * (i - 1) / 2);
        const float *rel = p.pos_ij + 3 * (p.edge_start[c] + (long long)i * n + j);
        const float rx = rel[0], ry = rel[1], rz = rel[2];
#pragma unroll
        for (int m = lane; m < NODES * UNIT / 4; m += 32) reinterpret_cast<float4 *>(hist)[m] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();

        const float x_end = (float)(NODES - PG_POINTS + 1);  // x below it: every node of the place exists
        const float d2_end = x_end * x_end / p.inv_h2 * 0.999999f;
        int count = 0;
        auto spread = [&]() {
            // x = d / h to a few 2^-24 of a node spacing, not of d: the square root of d2 / h^2 in two floats, one Newton step in
            // the remainder; kept as node and 24 bits of the rest
            const int longest = (__reduce_max_sync(FULL, count) + AT_ONCE - 1) / AT_ONCE * AT_ONCE;
            for (int t = 0; t < longest; ++t) {  // (shorter lists end in places beyond the nodes)
                const float d2 = __uint_as_float(list[t * 32 + lane]);
                const float s = d2 * p.inv_h2, s_low = fmaf(d2, p.inv_h2_low, fmaf(d2, p.inv_h2, -s));
                const float r = rsqrt_fast(fmaxf(s, 1e-30f)), x = s * r, fl = floorf(x);
                const float y = fmaf(0.5f * r, fmaf(-x, x, s) + s_low, x - fl);
                const int node = min((int)fl, NODES - PG_POINTS), rest = min(max(__float2int_rn(y * 0x1p24f), 0), 0xffffff);
                list[t * 32 + lane] = t < count ? ((unsigned)node << 24) | (unsigned)rest : (unsigned)NODES << 24;
            }
            __syncwarp();
#pragma unroll 1
            for (int from = 0; from < 4; ++from) {
                const int most = __reduce_max_sync(FULL, __shfl_sync(FULL, count, from * 8 + mine));
                const unsigned *at = list + from * 8 + mine;
#pragma unroll 1
                for (int t = 0; t < most; t += AT_ONCE, at += 32 * AT_ONCE) {  // AT_ONCE at a time: one's sums of products fill the other's waits
                    unsigned place[AT_ONCE];
                    float2 v[AT_ONCE][3], yy[AT_ONCE];
                    float y[AT_ONCE];
#pragma unroll
                    for (int w = 0; w < AT_ONCE; ++w) place[w] = at[32 * w];
#pragma unroll
                    for (int w = 0; w < AT_ONCE; ++w) {
                        y[w] = fmaf((float)(place[w] & 0xffffffu), 0x1p-24f, -0.5f);
                        yy[w] = make_float2(y[w] * y[w], y[w] * y[w]);
#pragma unroll
                        for (int q = 0; q < 3; ++q) v[w][q] = fma2(k[q][4], yy[w], k[q][3]);
                    }
#pragma unroll
                    for (int d = 2; d >= 0; --d)
#pragma unroll
                        for (int w = 0; w < AT_ONCE; ++w)
#pragma unroll
                            for (int q = 0; q < 3; ++q) v[w][q] = fma2(v[w][q], yy[w], k[q][d]);
#pragma unroll
                    for (int w = 0; w < AT_ONCE; ++w) {
                        float *node = hist + ((place[w] >> 24) + 3 * quarter) * UNIT + mine;
                        const float h0 = node[0], h1 = node[UNIT], h2 = node[2 * UNIT];
                        node[0] = h0 + fmaf(v[w][0].y, y[w], v[w][0].x);
                        node[UNIT] = h1 + fmaf(v[w][1].y, y[w], v[w][1].x);
                        node[2 * UNIT] = h2 + fmaf(v[w][2].y, y[w], v[w][2].x);
                        __syncwarp();  // (the next place may share nodes with this one, in another lane)
                    }
                }
            }
            count = 0;
        };
        int n1 = -R1, n2 = -R2 + quarter;
        while (n2 > R2) { n2 -= 2 * R2 + 1; ++n1; }
        while (__any_sync(FULL, n1 <= R1)) {
            const float f1 = (float)n1, f2 = (float)n2;
            const float bx = fmaf(cell.t2x, f2, fmaf(cell.t1x, f1, rx));
            const float by = fmaf(cell.t2y, f2, fmaf(cell.t1y, f1, ry));
            const float bz = fmaf(cell.t2z, f2, fmaf(cell.t1z, f1, rz));
            // no image of the column is closer than its line
            const float bt = fmaf(bz, cell.t3z, fmaf(by, cell.t3y, bx * cell.t3x));
            const float line2 = fmaf(bz, bz, fmaf(by, by, bx * bx)) - bt * bt * inv_t3sq;
            const bool in = n1 <= R1 && line2 * 0.9999f - 1e-6f < d2_end;
            if (__any_sync(FULL, in)) {
                auto image = [&](int n3) {
                    const float f3 = (float)n3;
                    const float dx = fmaf(cell.t3x, f3, bx), dy = fmaf(cell.t3y, f3, by), dz = fmaf(cell.t3z, f3, bz);
                    const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    list[count * 32 + lane] = __float_as_uint(d2);  // (stays where it counts)
                    count += in && n3 <= R3 && d2 < d2_end ? 1 : 0;
                };
                // (five images between two looks at the lists: the usual box's column)
                for (int n3 = -R3; n3 <= R3; n3 += ROOM) {
                    if (__any_sync(FULL, count >= LIST - ROOM)) spread();
#pragma unroll
                    for (int w = 0; w < ROOM; ++w) image(n3 + w);
                }
            }
            n2 += 4;
            while (n2 > R2) { n2 -= 2 * R2 + 1; ++n1; }
        }
        spread();
        // a pair without a finite distance: its rows must not come out as if it were not there
        const float probe = rx + ry + rz + cell.t1x + cell.t1y + cell.t1z + cell.t2x + cell.t2y + cell.t2z + cell.t3x + cell.t3y + cell.t3z;
        if (!(fabsf(probe) < 3e38f) && quarter == 0) hist[PG_BELOW * UNIT + mine] = __int_as_float(0x7fc00000);
        __syncwarp();

        // ---- out: a lane per pair and tile
        if (first + mine < pairs) {
            const long long slot = (variant == 0 ? (p.edge_start[c] + p.atom_start[c]) / 2 : info.z + (long long)(variant - 1) * pairs) + pair;
            uint4 *dst = reinterpret_cast<uint4 *>(p.grid.slots + slot * (64 * TILES));
            for (int t = quarter; t < TILES; t += 4) {
                const float *v = hist + t * PG_TILE * UNIT + mine;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    unsigned hi[4], lo[4];
#pragma unroll
                    for (int w = 0; w < 4; ++w) split_f16(v[(8 * half + 2 * w) * UNIT], v[(8 * half + 2 * w + 1) * UNIT], hi[w], lo[w]);
                    dst[t * 4 + half] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    dst[t * 4 + 2 + half] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
            }
        }
        __syncwarp();
    }
}

long long extra_slots(long long pairs) { return pairs / 2 + 8192; }

PairGrid carve(Carver &c, long long N, long long B, long long E, long long K)
{
    PairGrid g{};
    const long long pairs = (E + N) / 2;
    g.slot_count = pairs + extra_slots(pairs);
    g.counters = c.take<unsigned>(4 * (PG_LAYERS + 1));
    g.info = c.take<int4>((size_t)B);
    g.unit_start = c.take<int>((size_t)B + 1);
    g.tiles = c.take<int4>(2 * (size_t)(N / PG_ROWS + B));
    g.leftover = c.take<int>((size_t)N);
    g.basis = reinterpret_cast<uint4 *>(c.take<unsigned>(PG_BASIS_WORDS));
    g.basis_nodes = reinterpret_cast<uint4 *>(c.take<unsigned>(PG_BASIS_WORDS));
    g.projected = c.take<uint4>((size_t)PG_LAYERS * HEADS * PG_TILES_BASIS * 64);
    g.projected_scale = c.take<float>((size_t)PG_LAYERS * HEADS);
    g.slots = c.take<unsigned char>((size_t)g.slot_count * pg_slot_bytes(K));
    return g;
}

}  // namespace

size_t pair_grid_bytes(long long N, long long B, long long E, long long K)
{
    Carver c{nullptr};
    carve(c, N, B, E, K);
    return c.used;
}

PairGrid pair_grid_carve(void *memory, long long N, long long B, long long E, long long K)
{
    Carver c{static_cast<char *>(memory)};
    return carve(c, N, B, E, K);
}

// Whether vectors of these nodes serve the model: their range must cover an ordinary Gaussian (twice as narrow in variance as the
// widest) down to the floor, with 2 bits to spare; rows that need more are left over one by one.
bool pair_grid_params(long long K, double dist_max, double wscale, float a_widest, float floor_log2, PairGridParams &out)
{
    if (!(a_widest < 0.0f) || !(floor_log2 >= -40.0f) || !(K == 0 || (K == 64 && dist_max > 0 && wscale > 0))) return false;
    const double sigma_widest = sqrt(-0.5 / (double)a_widest);
    const double h = K > 0 ? (double)(float)dist_max / (double)K * (double)(float)wscale / 3.0 : 0.1 * sigma_widest;
    out.tiles = pg_tiles(K);
    out.inv_h2 = (float)(1.0 / (h * h));
    out.inv_h2_low = (float)(1.0 / (h * h) - (double)out.inv_h2);
    out.gauss = (float)(1.4426950408889634 * h * h);
    out.a_widest = a_widest;
    const double sigma_least = (K > 0 ? 9.0 : 5.0) * h;
    out.a_least = (float)(-0.5 / (sigma_least * sigma_least));
    out.floor_log2 = floor_log2;
    const double range = (out.tiles * PG_TILE - PG_POINTS) * h, need = sqrt(2.0 * 0.6931472 * (2.0 - floor_log2)) * sigma_widest * 0.7071068;
    return range >= need && sigma_least <= 0.75 * sigma_widest;
}

namespace {
void projections(PlanArgs &p, const PairAttn &b, const float *const *W, int W_stride, int calls)
{
    p.grid = b.grid;
    p.calls = calls;
    for (int c = 0; c < calls; ++c) p.W[c] = W[c * W_stride];
    p.wscale = (double)(float)b.wscale;
    p.wscale_f = (float)b.wscale;
    p.bits = (float)(-0.72134752044448170 / (9.0 * p.wscale * p.wscale));
}
}  // namespace

int launch_projected_basis(const PairAttn &b, const float *const *W, int W_stride, int calls, cudaStream_t s)
{
    PlanArgs p{};
    projections(p, b, W, W_stride, calls);
    projected_basis_kernel<<<calls * HEADS, 32 * PG_TILES_BASIS, 0, s>>>(p);
    return launch_status("projected_basis_kernel");
}

int launch_pair_grid_build(const PairAttn &b, const float *pos_ij, const float *tvecs, float a_widest, const float *const *W, int W_stride, int calls,
                           cudaStream_t s)
{
    PlanArgs p{};
    projections(p, b, W, W_stride, b.K > 0 && W != nullptr ? calls : 0);
    p.atom_start = b.atom_start; p.edge_start = b.edge_start; p.rvlen = b.rvlen; p.N = b.N; p.B = b.B; p.E = b.E;
    p.tile_cap = b.N / PG_ROWS + b.B; p.extra_cap = b.grid.slot_count - (b.E + b.N) / 2;
    p.rule = b.rule; p.a_widest = a_widest;
    p.basis_blocks = b.K > 0 && !b.projected ? (2 * PG_FRAGS * 32 + PLAN_THREADS - 1) / PLAN_THREADS : 0;
    pair_plan_kernel<<<1 + p.basis_blocks + p.calls * HEADS, PLAN_THREADS, 0, s>>>(p);
    BuildArgs a{};
    a.pos_ij = pos_ij; a.tvecs = tvecs; a.atom_start = b.atom_start; a.edge_start = b.edge_start; a.B = b.B; a.inv_h2 = b.par.inv_h2; a.inv_h2_low = b.par.inv_h2_low;
    a.grid = b.grid;
    auto kernel = b.K > 0 ? pair_grid_kernel<PG_TILES_BASIS> : pair_grid_kernel<PG_TILES_PLAIN>;
    const size_t smem = build_smem(b.par.tiles);
    static_assert(LIST % AT_ONCE == 0, "places at once");
    static_assert(build_smem(PG_TILES_BASIS) <= 48 * 1024, "no more shared memory than any kernel has");
    // (a crystal has at least one unit; those of the extra variants are not known here: the loop takes them)
    const long long units = ((b.E + b.N) / 2 + PG_UNIT - 1) / PG_UNIT + b.B, blocks = (units + BUILD_WARPS - 1) / BUILD_WARPS;
    const long long cap = (long long)sm_count() * BUILD_BLOCKS;
    kernel<<<(unsigned)(blocks < cap ? blocks : cap), 32 * BUILD_WARPS, smem, s>>>(a);
    return launch_status("pair_grid_kernel");
}

}  // namespace cf
