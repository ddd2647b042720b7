// Pair grids: the lattice sums of a batch as short vectors, one per pair of atoms, made once per batch for all layers.
//
// Every sum over the images of a pair (i, j) that an attention layer needs is of the form sum_n f(d_n) with f smooth on the
// scale of the radial basis: exp(a d^2) for the weights, exp(a d^2) g_k(d) for the basis sums, exp(a d^2) c(d) and
// exp(a d^2) d^2 in the backward.  The distances d_n belong to the geometry, f to the layer.  With nodes d_m of spacing h and
// interpolation weights L_q(y) that reproduce such functions from the POINTS nearest nodes,
//     sum_n f(d_n) = sum_m rho_m f(d_m),     rho_m = sum_n L_{m - floor(d_n / h)}(y_n)
// so the images enter once, in rho, and a layer evaluates its functions at the nodes only: two small matrix products per row
// instead of a sweep of its terms (3 to 1,000 images per pair).  rho_ij = rho_ji, so pairs i <= j are kept.
//
// Nodes: h is a third of the radial basis' standard deviation, twelve points.  The weights are the best ones for functions of
// a Gaussian spectrum of that width (simple kriging with its autocorrelation, conditional on y; polynomials of degree nine in
// y fit them to 1e-10).  For rows of random cells of 3-9 A the basis sums come out within 2.6e-8 (2-norm, arithmetic in 64
// bits) and the weights within 9e-9, a fraction of what float32 sums lose; ten points would give 1.8e-7, a spacing of
// 1 / 2.5 with fourteen points 5e-8, 1 / 4 with ten 9e-9 at a third more memory.  Without a basis the widths themselves set
// the scale: h = 0.1 of the widest standard deviation that the model can produce.
//
// Boxes: the cut-off rule gives every (atom, head) its own box of images, between the box of an infinitely narrow Gaussian and
// that of the widest.  A crystal has one set of vectors per box in that range (its variants: one for four cells of five, two
// for most others), and a head uses its own.
//
// A vector is stored as half-precision pairs (value, remainder), scaled by RHO_SCALE: per 16 nodes 32 bytes of values and 32
// of remainders, which is what the matrix instructions' operands are loaded from.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace cf {

constexpr int PG_POINTS = 12, PG_BELOW = 5;  // nodes floor(x) - 5 ... floor(x) + 6; node m sits at (m - 5) h
constexpr int PG_TILE = 16;                  // nodes per tile
constexpr int PG_TILES_BASIS = 11, PG_TILES_PLAIN = 5;
constexpr float PG_RHO_SCALE = 32.0f;
constexpr int PG_MAX_VARIANTS = 32;
constexpr int PG_UNIT = 8;                   // pairs of a unit of the build
constexpr int PG_ROWS = 8;                   // rows of a crystal that a block of the attention kernels takes
constexpr int PG_ALL_BOXES = 1 << 24;         // in PairGrid::info: the variants are all the boxes up to the widest Gaussian's
constexpr int PG_MAX_ATOMS = 64;             // (tables of eight rows in shared memory, two blocks per SM)
constexpr int PG_LAYERS = 32;                // calls per batch that find zeroed counters
// Grids lie where the batch would have its lists, and with a basis take more: 528 bytes per edge, lists and logits 300 (without one
// 240).  1,024 crystals of up to 60 atoms have a workspace of 923 MB for it, 649 MB with lists alone.  Beyond 16 M edges (thirteen
// times those crystals) a batch keeps its lists, so that no workspace is more than 4 GB larger for the grids.
constexpr size_t PG_MAX_BYTES = 8ull << 30;
constexpr long long PG_LEAST_EDGES = 5000, PG_LEAST_ROWS = 640;  // no smaller batch, no smaller training step goes this way

__host__ __device__ inline int pg_tiles(long long K) { return K > 0 ? PG_TILES_BASIS : PG_TILES_PLAIN; }
__host__ __device__ inline int pg_slot_bytes(long long K) { return 64 * pg_tiles(K); }

// Fragments of the matrix g_k(d_m) of the basis at the nodes, in halves (value, remainder) scaled by PG_BASIS_SCALE: per (node
// tile, bin tile) 32 lanes x (4 + 4) words; first with bins as rows, then with nodes as rows.
constexpr float PG_BASIS_SCALE = 16384.0f;
constexpr int PG_FRAGS = PG_TILES_BASIS * 4;
constexpr size_t PG_BASIS_WORDS = (size_t)PG_FRAGS * 32 * 8;

struct PairGrid {
    unsigned char *slots;        // vectors: pair (i <= j) of crystal c at (edge_start[c] + atom_start[c]) / 2 + its index
    int4 *info;                  // per crystal: smallest box (packed), variants per axis (packed), first extra slot, atoms
    int *unit_start;             // (B + 1): build units (PG_UNIT pairs of one variant) before a crystal
    int4 *tiles;                 // row tiles of the attention kernels: { crystal, first row, atoms (negative: no vectors), first
                                 // atom }, { first vector, first extra vector, smallest box, variants per axis }
    unsigned *counters;          // { tiles, units given out, -, - }, then per call { rows left over, ticket of their launch, -, - }
    int *leftover;               // rows left over by a call
    uint4 *basis;                // fragments, bins as rows
    uint4 *basis_nodes;          // fragments, nodes as rows
    uint4 *projected;            // W_h g(d_m) of every call: per (call, head, node tile) a fragment, channels as rows
    float *projected_scale;      // (call, head): what the products with them are divided by
    long long slot_count;
};
// Memory of a batch's grids and the offsets that only the model's entry points have.
struct GridMemory {
    void *memory;
    const int64_t *atom_start, *edge_start;
};
size_t encoder_lists_at(int64_t N, int64_t ff_dim);  // (encoder_forward.cu)
struct PairGridParams {
    int tiles;                   // node tiles of a vector
    float inv_h2, inv_h2_low;    // 1 / h^2 in two floats
    float gauss;                 // exp(a d_m^2) = 2^(a gauss (m - 5)^2)
    float a_widest;              // no layer has a wider Gaussian
    float a_least;               // rows with a narrower Gaussian (a below) are left over
    float floor_log2;
};

// Bytes for a batch, and whether a batch can go this way at all.
size_t pair_grid_bytes(long long N, long long B, long long E, long long K);
PairGrid pair_grid_carve(void *memory, long long N, long long B, long long E, long long K);
bool pair_grid_params(long long K, double dist_max, double wscale, float a_widest, float floor_log2, PairGridParams &out);
inline bool pair_grid_fits(long long N, long long B, long long E, long long max_atoms, long long K)
{
    return N > 0 && N < (1ll << 28) && max_atoms <= PG_MAX_ATOMS && E <= PG_MAX_ATOMS * N && pair_grid_bytes(N, B, E, K) <= PG_MAX_BYTES;
}
// What memory for batches of up to N atoms, B crystals and E edges holds for grids: those of any such batch, whether they are this
// one's or not (a batch that fits has at most 64 edges per atom), so that a workspace grows with each of its sizes.
inline size_t pair_grid_reserve(long long N, long long B, long long E, long long K)
{
    if (N <= 0 || E < PG_LEAST_EDGES) return 0;
    const size_t most = pair_grid_bytes(N, B, E < PG_MAX_ATOMS * N ? E : PG_MAX_ATOMS * N, K);
    return most < PG_MAX_BYTES ? most : PG_MAX_BYTES;
}
inline size_t pair_grid_reserve_training(long long N, long long B, long long E, long long K)
{
    return N < PG_LEAST_ROWS ? 0 : pair_grid_reserve(N, B, E > PG_LEAST_EDGES ? E : PG_LEAST_EDGES, K);
}
// Whether an inference batch gains by them.  The plan, the vectors and a block's fixed work (a row's Gaussians at the nodes, whatever
// its keys) want enough pairs and enough keys per row.  Times by row lists (without a basis: term lists), then over grids:
// - one forward at a time: 1, 4, 16, 64, 128 crystals of up to 30 atoms 211, 205, 218, 248, 354 us and 199, 200, 203, 220, 276; 1, 16,
//   64 of up to 60 182, 280, 462 and 216, 227, 273; 16, 64, 1,024 of up to 8 161, 182, 363 and 200, 199, 407; without a basis (seven
//   layers) 16, 64, 128 of up to 30 260, 316, 390 and 261, 285, 325, 16, 64 of up to 60 330, 503 and 288, 334;
// - sixteen batches in flight, where it is not latency that counts: 64, 128, 256 of up to 16 1,662, 1,876, 2,539 and 1,731, 2,075, 2,590;
//   16, 64, 128, 256 of up to 24 (16 keys per row) 1,924, 1,855, 2,459, 3,866 and 1,829, 1,853, 2,391, 3,389; 16, 64, 256 of up to
//   40 2,018, 3,166, 10,329 and 1,618, 2,355, 5,441; without a basis 64, 128, 256 of up to 24 2,080, 2,849, 4,566 and 2,248, 2,680,
//   3,673, 32 of up to 40 2,233 and 2,193, 256 of up to 16 (11 keys per row) 3,101 and 2,970.
// One line for all, so that a batch has the same bits however it is issued.
inline bool pair_grid_pays(long long N, long long B, long long E, long long max_atoms, long long K)
{
    if (!pair_grid_fits(N, B, E, max_atoms, K)) return false;
    return K > 0 ? (E >= PG_LEAST_EDGES && E >= 16 * N) || (E >= 30000 && E >= 11 * N) : E >= 20000 && E >= 11 * N;
}

// ... and whether a training step does: device time of a step (four layers), term lists against grids.  With a basis what it saves
// grows with the rows: 495, 653, 962, 1,271 rows (crystals of up to 30 or 40 atoms) 527, 657, 689, 926 us against 545, 596, 594,
// 685, few keys per row or many alike (1,173 rows of 6 keys 830 against 613, 504 of 41 650 against 630, 283 of 46 535 against 614).
// Without one a row by lists costs little: 653, 962, 1,271, 5,321 rows 521, 521, 642, 1,564 against 513, 501, 548, 1,200, and 1,693
// rows of 8 keys 576 against 584.
inline bool pair_grid_pays_training(long long N, long long B, long long E, long long max_atoms, long long K)
{
    return pair_grid_fits(N, B, E, max_atoms, K) && (K > 0 ? N >= PG_LEAST_ROWS && E >= 5 * N : N >= 960 && E >= 11 * N);
}

// One attention call over a batch's grids, and its backward.
struct PairAttn {
    const float *q, *k, *v, *a, *rvlen, *W;
    const int64_t *atom_start, *edge_start;
    long long N, B, E, K;
    int max_atoms;
    BoxRule rule;
    double dist_max, wscale;
    PairGridParams par;
    PairGrid grid;
    int call;
    float *out, *lse, *psi_row, *logit;  // psi_row, logit: or null
    unsigned char *left;         // per row: 1 if it was left over (or null)
    bool projected;              // the calls' projections at the nodes are made: no psi_row
    int *leftover;               // the rows, and their number in counters[4 (call + 1)]
    // backward
    const float *gout;
    float *gq, *gk, *gv, *ga, *glogit, *prob;
};
// The plan and the vectors (geometry, rule, sizes and parameters of `p`; a_widest: the widest Gaussian of any layer), and the basis at
// the nodes (for calls with psi_row) or, with p.projected, the calls' projections there: W of call c at W[c * W_stride], or by
// launch_projected_basis if W is null (a preparation that runs ahead of the weights' stream must not read them).
int launch_pair_grid_build(const PairAttn &p, const float *pos_ij, const float *tvecs, float a_widest, const float *const *W, int W_stride,
                           int calls, cudaStream_t s);
int launch_projected_basis(const PairAttn &p, const float *const *W, int W_stride, int calls, cudaStream_t s);
int launch_pair_attn_bwd(const PairAttn &p, cudaStream_t s);
int grid_attn_bwd_impl(const PairAttn &p, const float *pos_ij, const float *tvecs, const int64_t *batch, const int64_t *edges,
                       const int64_t *row_start, cudaStream_t s);
// The attention, and the rows that it leaves over by enumeration (their logits too, where p.logit is given).
int grid_attn_impl(const PairAttn &p, const float *pos_ij, const float *tvecs, const int64_t *batch, const int64_t *edges,
                   const int64_t *row_start, double cutoff_radius, int lattice_range, int minimum_range, cudaStream_t s);

}  // namespace cf
