// Dense products of an encoder layer boundary on the fifth-generation tensor cores (dense_tc.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "common.cuh"

namespace cf {

// Weight images.  A layer's projections are cut into 128 x 128 blocks; a block is 64 KB, the shared-memory image that
// the tensor instruction reads: the pieces h1 and h0 (tc5.cuh) one after the other, each two 64-deep k panels of 128 rows x
// 128 bytes with the 128-byte swizzle, so that a stage of the weight stream is one contiguous 32 KB copy of one piece, the
// small one first (Issuer::product).  Blocks are stored in the order in which the kernel consumes them; in front of them
// 1 KB of scales (float, 1 / s of every block).  The embedding has a third piece in front, so that an element's row comes
// out as the weight's column bit for bit.
constexpr int TC_PIECE_BYTES = 32768;
constexpr int TC_BLOCK_BYTES = 2 * TC_PIECE_BYTES;
constexpr int TC_HEADER_BYTES = 1024;
constexpr int TC_EMBED_PIECES = 3;
constexpr size_t TC_EMBED_BYTES = TC_HEADER_BYTES + TC_EMBED_PIECES * TC_PIECE_BYTES;
inline size_t tc_image_bytes(int blocks) { return (size_t)TC_HEADER_BYTES + (size_t)blocks * TC_BLOCK_BYTES; }
inline int tc_tail_blocks(int ff) { return 1 + 2 * (ff / 128); }  // Wo, then W1 / W2 chunks interleaved
inline int tc_layer_blocks(int ff) { return tc_tail_blocks(ff) + 3; }

// One block to pack: element (n, k) is src[n ld + k] (or src[k ld + n] with trans), zero outside rows x cols; the scale
// is that of the largest magnitude among `group` arrays of group_elems values each.
struct PackBlock {
    const float *src, *group[3];
    int group_elems, ld;
    short rows, cols, trans, block;   // block: index in the image
    int pieces;
    unsigned char *image;
};
constexpr int PACK_MAX = 56;                          // blocks of one launch (the job is a kernel parameter)
constexpr int TC_MAX_FF = 128 * ((PACK_MAX - 4) / 2);  // a layer is packed by one launch
struct PackJob {
    PackBlock b[PACK_MAX];
};
int launch_pack(const PackJob &job, int count, cudaStream_t s);
// The blocks of one layer, forward order: [Wo, W1_0, W1_1, W2_0, W1_2, W2_1, ..., Wq, Wk, Wv].  Appends to job.
void pack_layer_forward(PackJob &job, int &count, unsigned char *image, int ff, const float *Wq, const float *Wk, const float *Wv,
                        const float *Wo, const float *W1, const float *W2);
void pack_embedding(PackJob &job, int &count, unsigned char *image, const float *W, int feature_dim);

struct DenseForward {
    long long N;
    int ff;
    bool chained, weights_fresh;    // weights_fresh: the images were written earlier on this stream by a kernel that may still run
    // tail of the layer whose attention just ran (image null: none)
    const unsigned char *tail;
    const float *attn, *bo, *b1, *b2;
    // embedding (only without a tail): x = features W^T
    const unsigned char *embed;
    const float *features;
    const int64_t *species;
    int feature_dim;
    // head of the next layer (image null: none)
    const unsigned char *head;
    const float *bqkv, *w_pos;
    float gauss_scale, gauss_shift, a_factor, elu_beta, lower_bound;
    float a_factor_hi, lower_bound_hi;  // heads 4-7 (domain "multihead": the reciprocal-space half; else as heads 0-3)
    bool inverse;                       // a = a_factor / f instead of a_factor f (domain "RECI")
    // activations
    const float *x_in;   // (N,128) features the tail's residual (or, without tail and embedding, the head) reads
    float *x_out;        // (N,128) features after the tail / embedding
    float *q, *k, *v, *a;
    float *y_save, *h_save;  // training: y (N,128) and the hidden units (N, ff), or null
    unsigned *status;        // (set by the launch: wait_status)
};

// The packed-weight pointers of the one-call forwards (slot 10 of a layer, W_embed_packed) carry bit 0 set when they name
// such an image rather than fragments for the warp-level dense block (dense_block.cu).
inline bool is_tc_image(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 1) != 0; }
inline const unsigned char *tc_image(const void *p) { return reinterpret_cast<const unsigned char *>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)1); }
inline bool dense_tc_images(int num_layers, const float *const *weights)
{
    bool all = num_layers > 0;
    for (int l = 0; l < num_layers; ++l) all = all && is_tc_image(weights[11 * l + 10]);
    return all;
}

int launch_dense_forward(const DenseForward &p, cudaStream_t s);

// A forward whose first boundary (embedding and the first layer's head) has been launched ahead of the rest, with what it
// wrote; head_stage carves it from N (4 x 128 + 8) floats.
struct HeadStage {
    float *x, *q, *k, *v, *a;
    void *event;  // after which it has been written
};
inline HeadStage head_stage(float *memory, long long N, void *event)
{
    HeadStage h;
    h.event = event;
    h.x = memory; h.q = h.x + N * 128; h.k = h.q + N * 128; h.v = h.k + N * 128; h.a = h.v + N * 128;
    return h;
}
// head of a layer (11 weight pointers, 6 scalars, as in cf_encoder_forward)
inline void dense_head_of(DenseForward &d, const float *const *w, const double *sc)
{
    d.head = tc_image(w[10]); d.bqkv = w[1]; d.w_pos = w[2];
    d.gauss_scale = (float)sc[0]; d.gauss_shift = (float)sc[1]; d.a_factor = (float)sc[2];
    d.elu_beta = (float)sc[3]; d.lower_bound = (float)sc[4];
    d.a_factor_hi = d.a_factor; d.lower_bound_hi = d.lower_bound;
}
// Host read of a batch's sizes beside the work that `launch` queues on the side stream (encoder_forward.cu).
int read_sizes_beside(const int64_t *sizes, int64_t B, int64_t *counts, cudaStream_t s, int (*launch)(void *, cudaStream_t), void *arg,
                      void **begun_event);
int join_begun(void *begun_event, cudaStream_t s);

// ---- training (dense_tc_bwd.cu) ---------------------------------------------------------------------------------------
// The blocks of one layer in the backward kernel's order, every one transposed: [Wq, Wk, Wv] and
// [W2_0, W2_1, W1_0, W2_2, W1_1, ..., Wo].  Appends to job.
void pack_layer_backward(PackJob &job, int &count, unsigned char *image, int ff, const float *Wq, const float *Wk, const float *Wv,
                         const float *Wo, const float *W1, const float *W2);

// Backward of a boundary: the head of layer l + 1, then the tail of layer l.
struct DenseBackward {
    long long N;
    int ff;
    // head (image null: none): gx = g_res + gq' Wq + gk Wk + gv Wv, gq' = gq / 4 + galpha w_pos
    const unsigned char *head;
    const float *q, *w_pos;      // the saved query (scaled by 1/4)
    float gauss_scale, gauss_shift, a_factor, elu_beta, lower_bound, a_factor_hi, lower_bound_hi;  // as in DenseForward
    bool inverse;
    float *gq, *ga;              // in: gradients of the scaled query and of a; out: gq' and galpha
    const float *gk, *gv, *g_res;
    float *gx;                   // (N,128) out (with a head), in (without)
    // tail (image null: none): gh = (gx W2) [h > 0], gy = gx + gh W1, gattn = gy Wo
    const unsigned char *tail;
    const float *h;              // (N, ff) the saved hidden units
    float *gh, *gy, *gattn;
    unsigned *status;            // (set by the launch: wait_status)
};
int launch_dense_backward(const DenseBackward &p, cudaStream_t s);

// One 128 x 128 block of a weight gradient: out[i ld + j] = sum_n g[n ldg + i] x[n ldx + j] (j < cols), and, where bias is
// not null, bias[i] = sum_n g[n ldg + i].
struct GradJob {
    const float *g, *x;
    long long rows;
    int ldg, ldx, x_cols, ldo;
    float *out, *bias;
};
constexpr int GRAD_MAX = 56;            // jobs of one launch (a kernel parameter)
constexpr int GRAD_MAX_SPLITS = 16;
constexpr int GRAD_PARTIAL = 128 * 128 + 128;
struct GradJobs {
    GradJob j[GRAD_MAX];
};
// Launches the jobs with the rows split so that the blocks fill the SMs; partial holds grad_partial_floats(count, rows of
// job 0).
size_t grad_partial_floats(int count, long long rows);
int launch_weight_grads(const GradJobs &jobs, int count, float *partial, cudaStream_t s);

}  // namespace cf
