// Term lists (see term_list.cuh): the build kernel and phi from a list.
#include "lattice_core.cuh"
#include "term_list.cuh"

namespace cf {
namespace {

constexpr int TL_WARPS = 8;

// The translations that the list of a key can hold: its box n_lo .. n_lo + w - 1, the bounding box of the ball
// |r + n T|^2 <= threshold clipped to the rule's box.  With b_i the reciprocal rows (b_i . t_j = delta_ij),
// (r + n T) . b_i = s_i + n_i and |x . b_i| <= |x| |b_i| bound every digit: |n_i + s_i| <= rho |b_i|, s_i = r . b_i,
// rho = sqrt(threshold); widened a little beyond any rounding (the test on d2 decides membership).
struct CellDual {
    float b1x, b1y, b1z, b2x, b2y, b2z, b3x, b3y, b3z, l1, l2, l3;
    bool prune;  // false: a flat cell keeps the whole box
    __device__ __forceinline__ void init(const Cell &c)
    {
        const float c1x = c.t2y * c.t3z - c.t2z * c.t3y, c1y = c.t2z * c.t3x - c.t2x * c.t3z, c1z = c.t2x * c.t3y - c.t2y * c.t3x;
        const float c2x = c.t3y * c.t1z - c.t3z * c.t1y, c2y = c.t3z * c.t1x - c.t3x * c.t1z, c2z = c.t3x * c.t1y - c.t3y * c.t1x;
        const float c3x = c.t1y * c.t2z - c.t1z * c.t2y, c3y = c.t1z * c.t2x - c.t1x * c.t2z, c3z = c.t1x * c.t2y - c.t1y * c.t2x;
        const float det = c.t1x * c1x + c.t1y * c1y + c.t1z * c1z;
        prune = fabsf(det) > 1e-12f;
        const float i = prune ? 1.0f / det : 0.0f;
        b1x = c1x * i; b1y = c1y * i; b1z = c1z * i;
        b2x = c2x * i; b2y = c2y * i; b2z = c2z * i;
        b3x = c3x * i; b3y = c3y * i; b3z = c3z * i;
        l1 = sqrtf(b1x * b1x + b1y * b1y + b1z * b1z); l2 = sqrtf(b2x * b2x + b2y * b2y + b2z * b2z); l3 = sqrtf(b3x * b3x + b3y * b3y + b3z * b3z);
    }
};
__device__ __forceinline__ void digit_range(float rho, float len, float s, int R, int &lo, int &hi)
{
    const float m = rho * len + 1e-3f;
    // (clamped as floats first: the conversions then see small values only)
    lo = (int)ceilf(fmaxf(-m - s, (float)-R));
    hi = (int)floorf(fminf(m - s, (float)R));
}

// One warp per row, one key per lane, or several lanes where the row has few keys (they deal the columns of the key's box
// among themselves).  Threshold, box and terms of a key are its lanes' own work (two walks of the box, to count and to
// fill); the offsets of a chunk of keys come from a scan over the lanes.  A box holds about twice the
// listed terms, whatever the cell: the walk of the rule's box by columns that this replaces took 0.53 ms for 64 crystals
// of 100-200 atoms (1.5 M edges, 3 terms each), this one 0.15 ms.
__global__ void __launch_bounds__(32 * TL_WARPS) term_list_build_kernel(const TermListBuild p)
{
    const int lane = threadIdx.x & 31;
    const bool near27 = p.rule.cutoff == 0.0f ? true : p.rule.minimum_range >= 1;
    for (long long slot = (long long)blockIdx.x * TL_WARPS + (threadIdx.x >> 5); slot < p.N; slot += (long long)gridDim.x * TL_WARPS) {
        const long long i = p.row_order ? p.row_order[slot] : slot;
        const long long c = p.batch[i];
        const long long e0 = p.row_start[i];
        const int n = (int)(p.row_start[i + 1] - e0);
        if (n > p.max_atoms) {  // the caller understated max_atoms: no list, the row kernel poisons the row
            for (int j = lane; j < n; j += 32) p.start[e0 + j] = -1;
            continue;
        }
        Cell cell;
        cell.load(p.tvecs + 9 * c);
        CellDual dual;
        dual.init(cell);
        float rvl[3] = {0.f, 0.f, 0.f};
        if (p.rvlen) { rvl[0] = p.rvlen[3 * c]; rvl[1] = p.rvlen[3 * c + 1]; rvl[2] = p.rvlen[3 * c + 2]; }
        const int pk = packed_box(p.rule, p.a_widest, p.rvlen ? rvl : nullptr);  // contains every head's box
        const int R1 = box_r1(pk), R2 = box_r2(pk), R3 = box_r3(pk);
        // the lane's key: position, threshold (an upper bound of the smallest squared distance ANY head's box can contain,
        // plus the window; boxes of half-width >= 1 contain the 27 nearest translations, otherwise only n = 0 is certain),
        // and visit(d2, n1, n2, n3) for every listed term
        const int lanes = n > 16 ? 1 : n > 8 ? 2 : n > 4 ? 4 : n > 2 ? 8 : n > 1 ? 16 : 32;  // of a key
        const int sub = lane & (lanes - 1), first_key = lane / lanes;
        auto threshold = [&](float rx, float ry, float rz) {
            float m = fmaf(rz, rz, fmaf(ry, ry, rx * rx));
            auto image = [&](float f1, float f2, float f3) {
                const float dx = fmaf(cell.t3x, f3, fmaf(cell.t2x, f2, fmaf(cell.t1x, f1, rx)));
                const float dy = fmaf(cell.t3y, f3, fmaf(cell.t2y, f2, fmaf(cell.t1y, f1, ry)));
                const float dz = fmaf(cell.t3z, f3, fmaf(cell.t2z, f2, fmaf(cell.t1z, f1, rz)));
                m = fminf(m, fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
            };
            if (near27 && R1 > 0 && R2 > 0 && R3 > 0) {  // (unrolled: independent terms, nine at a time)
#pragma unroll 1
                for (int n1 = -1; n1 <= 1; ++n1)
#pragma unroll
                    for (int t = 0; t < 9; ++t) image((float)n1, (float)(t / 3 - 1), (float)(t % 3 - 1));
            } else if (near27) {
                for (int n1 = -min(R1, 1); n1 <= min(R1, 1); ++n1)
                    for (int n2 = -min(R2, 1); n2 <= min(R2, 1); ++n2)
                        for (int n3 = -min(R3, 1); n3 <= min(R3, 1); ++n3) image((float)n1, (float)n2, (float)n3);
            }
            return m + p.window;
        };
        auto walk_key = [&](float rx, float ry, float rz, float thr, auto &&visit) {
            int lo1 = -R1, hi1 = R1, lo2 = -R2, hi2 = R2, lo3 = -R3, hi3 = R3;
            if (dual.prune) {
                const float rho = sqrtf(fmaxf(thr, 0.f)) * 1.0001f;
                digit_range(rho, dual.l1, rx * dual.b1x + ry * dual.b1y + rz * dual.b1z, R1, lo1, hi1);
                digit_range(rho, dual.l2, rx * dual.b2x + ry * dual.b2y + rz * dual.b2z, R2, lo2, hi2);
                digit_range(rho, dual.l3, rx * dual.b3x + ry * dual.b3y + rz * dual.b3z, R3, lo3, hi3);
            }
            const int w2 = hi2 - lo2 + 1;
            if (w2 <= 0) return;
            int n1 = lo1, n2 = lo2 + sub;
            while (n2 > hi2) { n2 -= w2; ++n1; }
            while (n1 <= hi1) {
                // r + n1 t1 + n2 t2 + n3 t3, contracted like the reference's expression
                const float f1 = (float)n1, f2 = (float)n2;
                const float ex = fmaf(cell.t2x, f2, fmaf(cell.t1x, f1, rx));
                const float ey = fmaf(cell.t2y, f2, fmaf(cell.t1y, f1, ry));
                const float ez = fmaf(cell.t2z, f2, fmaf(cell.t1z, f1, rz));
#pragma unroll 2
                for (int n3 = lo3; n3 <= hi3; ++n3) {
                    const float f3 = (float)n3;
                    const float dx = fmaf(cell.t3x, f3, ex), dy = fmaf(cell.t3y, f3, ey), dz = fmaf(cell.t3z, f3, ez);
                    const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    if (d2 <= thr) visit(d2, n1, n2, n3);
                }
                n2 += lanes;
                while (n2 > hi2) { n2 -= w2; ++n1; }
            }
        };
        // ---- count (a key's threshold waits in its dmin for the second walk)
        int total = 0, own = 0;  // own: terms of this lane, where a key has several lanes (the row is one chunk then)
        for (int j0 = 0; j0 < n; j0 += 32) {
            const int j = j0 + first_key;
            int cnt = 0;
            float thr = 0.f;
            if (j < n) {
                const float *pp = p.pos_ij + 3 * (e0 + j);
                thr = threshold(pp[0], pp[1], pp[2]);
                walk_key(pp[0], pp[1], pp[2], thr, [&](float, int, int, int) { ++cnt; });
            }
            own = cnt;
            total += cnt;
            for (int o = 1; o < lanes; o <<= 1) cnt += __shfl_xor_sync(FULL, cnt, o);
            if (j < n && sub == 0) {
                p.count[e0 + j] = cnt;
                p.dmin[e0 + j] = thr;
            }
        }
        __syncwarp();  // (the other lanes of a key read its threshold)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(FULL, total, o);
        long long base = 0;
        if (lane == 0) {
            const unsigned long long at = atomicAdd(p.cursor, (unsigned long long)total);
            base = (at + (unsigned long long)total <= (unsigned long long)p.capacity && at + (unsigned long long)total < (1ull << 31)) ? (long long)at : -1;
        }
        base = __shfl_sync(FULL, base, 0);
        if (base < 0) {  // the pool is full: this row is processed by enumeration
            for (int j = lane; j < n; j += 32) p.start[e0 + j] = -1;
            continue;
        }
        // ---- fill, keys ascending
        long long run = base;
        for (int j0 = 0; j0 < n; j0 += 32) {
            const int j = j0 + first_key;
            const int cnt = j >= n ? 0 : lanes > 1 ? own : p.count[e0 + j];  // (this lane's own store)
            const float thr = j < n ? p.dmin[e0 + j] : 0.f;
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += up;
            }
            float dm = INFINITY;
            if (j < n) {
                const long long first = run + incl - cnt;
                if (sub == 0) p.start[e0 + j] = (int)first;
                float2 *out = p.pool + first;
                const float *pp = p.pos_ij + 3 * (e0 + j);
                walk_key(pp[0], pp[1], pp[2], thr, [&](float d2, int n1, int n2, int n3) {
                    *out++ = make_float2(d2, __int_as_float(pack_key(j, abs(n1), abs(n2), abs(n3))));
                    dm = fminf(dm, d2);
                });
            }
            for (int o = 1; o < lanes; o <<= 1) dm = fminf(dm, __shfl_xor_sync(FULL, dm, o));
            if (j < n && sub == 0) p.dmin[e0 + j] = dm;
            run += __shfl_sync(FULL, incl, 31);
        }
    }
}

// TPE (1, 2, 4 or 8) lanes per edge: phi of all heads from the edge's entries (boxes applied per head).  The lanes of
// a group split the eight box computations, read the entries sub, sub + TPE, ... (the group's loads are contiguous)
// and keep partial sums for all heads, combined by a fixed butterfly.  Few lanes per edge for batches of many edges
// with short lists (large cells), eight for few edges with long lists (small cells).  Rows without a list, and edges
// where a head's box misses every listed term, take the enumerating code.
template <int TPE>
__global__ void __launch_bounds__(128) phi_from_list_kernel(const PhiListArgs p)
{
    const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gtid == 0 && p.zero_word) *p.zero_word = 0u;
    const long long e_raw = gtid / TPE;
    const int sub = (int)(gtid % TPE);
    const bool live = e_raw < p.E;
    const long long e = live ? e_raw : p.E - 1;  // idle tail lanes shadow the last edge so that shuffles stay full
    const long long i = p.edges[e];
    const long long c = p.batch[i];
    float rvl[3] = {0.f, 0.f, 0.f};
    if (p.rvlen) { rvl[0] = p.rvlen[3 * c]; rvl[1] = p.rvlen[3 * c + 1]; rvl[2] = p.rvlen[3 * c + 2]; }
    constexpr int PER = 8 / TPE;  // heads whose box this lane computes
    const int lane = threadIdx.x & 31, group0 = lane & ~(TPE - 1);
    float a_mine[PER];
    int pk_mine[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        a_mine[u] = p.a[i * HEADS + sub * PER + u];
        pk_mine[u] = packed_box(p.rule, a_mine[u], p.rvlen ? rvl : nullptr);
    }
    float a[8], a2[8];
    int pk[8];
    float a2max = -INFINITY;
#pragma unroll
    for (int h = 0; h < 8; ++h) {
        a[h] = __shfl_sync(FULL, a_mine[h % PER], group0 + h / PER);
        pk[h] = __shfl_sync(FULL, pk_mine[h % PER], group0 + h / PER);
        a2[h] = a[h] * LOG2E;
        a2max = fmaxf(a2max, a2[h]);
    }
    float z[8];
    const int first = p.list.start[e];
    const int cnt = first >= 0 ? p.list.count[e] : 0;
    const float m = first >= 0 ? p.list.dmin[e] : 0.f;
    const float2 *ent = p.list.pool + (first >= 0 ? first : 0);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // four entries per step, the next four requested meanwhile: the lists stream from memory, and a step is short
    const float2 none = make_float2(INFINITY, 0.f);
    float2 nx[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) nx[u] = sub + u * TPE < cnt ? __ldg(ent + sub + u * TPE) : none;
    for (int t = sub; t < cnt; t += 4 * TPE) {
        float2 en[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            en[u] = nx[u];
            nx[u] = t + (4 + u) * TPE < cnt ? __ldg(ent + t + (4 + u) * TPE) : none;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float rel = en[u].x - m;
            if (a2max * rel < p.floor_log2) continue;  // below the floor for every head (or no entry)
            const int bytes = key_bytes(__float_as_int(en[u].y));
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                const float w = ex2(a2[h] * rel);
                s[h] += bytes_in_box(bytes, pk[h]) ? w : 0.f;
            }
        }
    }
    bool done = cnt > 0;
#pragma unroll
    for (int h = 0; h < 8; ++h) {  // (all lanes of the warp take part in the shuffles, listed or not)
        float t = s[h];
#pragma unroll
        for (int o = 1; o < TPE; o <<= 1) t += __shfl_xor_sync(FULL, t, o);
        z[h] = fmaf(m, a[h], logf(t));
        done = done && t > 1e-30f;  // a head whose box misses the listed terms: enumerate instead
    }
    if (!done && sub == 0) {
        Cell cell;
        cell.load(p.tvecs + 9 * c);
        edge_phi<1>(p.rule, a, p.rvlen ? p.rvlen + 3 * c : nullptr, cell, p.pos_ij[3 * e], p.pos_ij[3 * e + 1],
                    p.pos_ij[3 * e + 2], p.floor_log2, 0, z);
    }
    if (live && sub == 0) {
        float4 *zo = reinterpret_cast<float4 *>(p.z + e * HEADS);
        zo[0] = make_float4(z[0], z[1], z[2], z[3]);
        zo[1] = make_float4(z[4], z[5], z[6], z[7]);
    }
}

}  // namespace

// About 25 entries per edge are needed for cells of 3-15 Angstrom edges at the default widths (sphere of the window
// over the cell volume), 3 for cells of 10-25 Angstrom; rows that do not fit are enumerated instead.
size_t term_pool_entries(long long N, long long E) { return (size_t)(32 * E + 64 * N + (1ll << 20)); }

size_t term_list_workspace_bytes(long long N, long long E)
{
    return sizeof(int) * (3 * (size_t)E + 32) + sizeof(float2) * term_pool_entries(N, E);
}

void term_list_carve(void *workspace, long long N, long long E, int **start, int **count, float **dmin,
                     unsigned long long **cursor, float2 **pool)
{
    (void)N;
    auto align = [](const void *ptr, uintptr_t to) { return (reinterpret_cast<uintptr_t>(ptr) + to - 1) & ~(to - 1); };
    int *dir = static_cast<int *>(workspace);
    *start = dir;
    *count = dir + E;
    *dmin = reinterpret_cast<float *>(dir + 2 * E);
    *cursor = reinterpret_cast<unsigned long long *>(align(dir + 3 * E, 8));
    *pool = reinterpret_cast<float2 *>(align(dir + 3 * E + 8, 16));
}

int launch_term_list_build(const TermListBuild &b, cudaStream_t s)
{
    if (b.N == 0) return CF_OK;
    if (cudaMemsetAsync(b.cursor, 0, sizeof(unsigned long long), s) != cudaSuccess) return launch_status("term list cursor");
    const long long want = (b.N + TL_WARPS - 1) / TL_WARPS, cap = (long long)sm_count() * 8;
    term_list_build_kernel<<<(unsigned)(want < cap ? want : cap), 32 * TL_WARPS, 0, s>>>(b);
    return launch_status("term_list_build_kernel");
}

int launch_phi_from_list(const PhiListArgs &p, cudaStream_t s)
{
    if (p.E == 0) return CF_OK;
    // lanes per edge: as many as keep the grid at about a wave's threads (a wave costs its loads of edge, atom, crystal and
    // widths, about 3 us, whatever the lists hold: 141,000 edges took 45 us per call with eight lanes, 31 with two)
    const long long per_wave = (long long)sm_count() * 2048;
    const int tpe = p.E * 8 <= per_wave ? 8 : (p.E * 4 <= per_wave ? 4 : (p.E * 2 <= per_wave ? 2 : 1));
    const unsigned blocks = (unsigned)((p.E * tpe + 127) / 128);
    switch (tpe) {
        case 8: phi_from_list_kernel<8><<<blocks, 128, 0, s>>>(p); break;
        case 4: phi_from_list_kernel<4><<<blocks, 128, 0, s>>>(p); break;
        case 2: phi_from_list_kernel<2><<<blocks, 128, 0, s>>>(p); break;
        default: phi_from_list_kernel<1><<<blocks, 128, 0, s>>>(p); break;
    }
    return launch_status("phi_from_list_kernel");
}

}  // namespace cf

extern "C" int64_t cf_term_list_workspace_bytes(int64_t N, int64_t E)
{
    return (int64_t)cf::term_list_workspace_bytes(N, E);
}

extern "C" int cf_term_list_build(const float *pos_ij, const float *tvecs, const float *rvlen, const int64_t *batch,
                                  const int64_t *edges, const int64_t *row_start, const int32_t *row_order, int64_t N,
                                  int64_t E, int64_t max_atoms, double cutoff_radius, int lattice_range,
                                  int minimum_range, double a_widest, void *workspace, void *stream)
{
    using namespace cf;
    CF_REQUIRE(N >= 0 && E >= 0, CF_ERR_INVALID, "cf_term_list_build: negative size");
    CF_REQUIRE(a_widest < 0, CF_ERR_INVALID, "cf_term_list_build: a_widest must be negative");
    CF_REQUIRE(max_atoms >= 1 && max_atoms <= 2048, CF_ERR_RANGE, "cf_term_list_build: max_atoms=%lld outside [1,2048]",
               (long long)max_atoms);
    CF_REQUIRE(lattice_range >= 0 && lattice_range <= CF_MAX_RANGE && minimum_range >= 0, CF_ERR_RANGE,
               "cf_term_list_build: lattice_range %d outside [0,%d]", lattice_range, CF_MAX_RANGE);
    if (N == 0) return CF_OK;
    CF_REQUIRE(pos_ij && tvecs && batch && edges && row_start && workspace, CF_ERR_INVALID, "cf_term_list_build: null pointer");
    TermListBuild tb{};
    tb.pos_ij = pos_ij; tb.tvecs = tvecs; tb.rvlen = cutoff_radius != 0.0 ? rvlen : nullptr;
    tb.batch = batch; tb.edges = edges; tb.row_start = row_start; tb.row_order = row_order;
    tb.N = N; tb.E = E; tb.max_atoms = (int)max_atoms;
    tb.rule = BoxRule{(float)cutoff_radius, lattice_range, minimum_range};
    tb.a_widest = (float)a_widest;
    tb.window = term_window(weight_floor_log2(), (float)a_widest);
    term_list_carve(workspace, N, E, &tb.start, &tb.count, &tb.dmin, &tb.cursor, &tb.pool);
    tb.capacity = (long long)term_pool_entries(N, E);
    return launch_term_list_build(tb, as_stream(stream));
}
