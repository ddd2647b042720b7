// Attention forward by blocks of eight rows (infinite_attn_block.cu).
#pragma once
#include "common.cuh"
#include "term_list.cuh"

namespace cf {

// Largest crystal the kernel takes: two blocks with their tables of 8 rows x 8 heads per key fit one SM.
constexpr int ROW_BLOCK_MAX_ATOMS = 200;
// Batches of smaller crystals keep the row kernel: their cells are small too, a row of a dense one lists thousands of
// terms, and here a row is one warp's (256 crystals of up to 40 atoms: 0.28 ms per call against 0.21 ms).
constexpr int ROW_BLOCK_MIN_ATOMS = 64;
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
