// Attention forward by blocks of eight rows (infinite_attn_block.cu).
#pragma once
#include "common.cuh"
#include "term_list.cuh"

namespace cf {

// Largest crystal the kernel takes: two blocks with their tables of 8 rows x 8 heads per key fit one SM (asserted beside the
// kernel).
constexpr int ROW_BLOCK_MAX_ATOMS = 210;
// Batches of smaller crystals keep the row kernel: their cells are small too, a row of a dense one lists thousands of
// terms, and here a row is one warp's (256 crystals of up to 40 atoms: 0.28 ms per call against 0.21 ms).
constexpr int ROW_BLOCK_MIN_ATOMS = 64;
// Whether a batch goes by blocks.  All its rows do or none, so it needs
// - enough rows that the blocks of eight have most of the SMs to themselves: below five rows per SM the row kernel, with a
//   block per row, is faster (forward of 1, 4, 6, 12 crystals of 150 atoms by rows 327, 477, 524, 768 us, by blocks 401, 450,
//   442, 479; of 200 atoms 357, 571, 699, 962 against 521, 531, 564, 794);
// - not mostly small crystals, whose dense cells make long rows: at 32 atoms per crystal on average the two are even (64, 128,
//   255 crystals of 1-40 atoms with 8, 16, 32 of 100-200, 35 on average: by rows 752, 1,170, 2,224 us, by blocks 854, 1,094,
//   1,974; 64, 255 with 4, 16, 28 on average: 647, 1,611 against 820, 1,651; with one: 539, 1,123 against 786, 1,369; 60 of 66
//   atoms: 813 against 526).
// What the cells hold is not known here: 60 crystals of 66 atoms in the cells of 3-15 A of small ones take 1,176 us by rows and
// 1,606 by blocks, in cells of 10-25 A 813 and 526.
inline bool by_row_blocks(long long N, long long B, long long max_atoms)
{
    return max_atoms > ROW_BLOCK_MIN_ATOMS && max_atoms <= ROW_BLOCK_MAX_ATOMS && N >= 5ll * sm_count() && N >= 32 * B && N < (1ll << 31);
}
constexpr int ROW_BLOCK_LAYERS = 32;  // calls per batch that find a zeroed scheduling block

// Scheduling memory of a batch: the blocks' first atoms, the rows left over, and counters { blocks, -, -, - }, then per call
// { ticket, rows left over, ticket of the left-over launch, - }.
struct RowBlocks {
    int *blocks, *leftover;
    unsigned *counters;
};
inline size_t row_blocks_words(long long N) { return 2 * (size_t)N + 4 * (ROW_BLOCK_LAYERS + 1) + 8; }
inline RowBlocks row_blocks_carve(void *memory, long long N)
{
    RowBlocks b;
    b.counters = static_cast<unsigned *>(memory);
    b.blocks = static_cast<int *>(memory) + 4 * (ROW_BLOCK_LAYERS + 1);
    b.leftover = b.blocks + N;
    return b;
}
// Zeroes the counters and lists the blocks (after the batch's geometry, on the same stream).
int launch_row_blocks(const RowBlocks &b, const int32_t *row_order, const int64_t *row_start, const int64_t *edges, long long N, long long E,
                      cudaStream_t s);
// One attention call; `call` < ROW_BLOCK_LAYERS: a different one for every call of the batch.
int block_attn_impl(const float *q, const float *k, const float *v, const float *a, const float *pos_ij, const float *tvecs,
                    const float *rvlen, const int64_t *batch, const int64_t *edges, const int64_t *row_start, int64_t N, int64_t B,
                    int64_t E, int64_t K, int64_t max_atoms, double dist_max, double wscale, const float *W, double cutoff_radius,
                    int lattice_range, int minimum_range, float *out, float *logit, float *lse, float *psi_row, const TermList &list,
                    const RowBlocks &blocks, int call, cudaStream_t s);

}  // namespace cf
