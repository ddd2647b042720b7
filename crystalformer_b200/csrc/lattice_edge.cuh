// One warp, one edge: the parts the forward and backward lattice-sum kernels share.
//
// A warp's edge is a few hundred instructions, so two things decide its cost: the dependent loads in front of it (edge ->
// atom -> crystal -> lattice), and what is spent on the translations that turn out not to matter.  EdgeStream fetches the
// constants of the next edges while the current one is processed, one word per lane.  BoxWalk enumerates the translation
// box with the digits of the common 5 x 5 x 5 box in registers; only d2 is computed for every translation, those within
// reach of the widest head are collected in shared memory (EdgeTerms), and the eight exponentials are spent on full
// warps of collected terms.
#pragma once
#include "lattice_core.cuh"

namespace cf {

// The constants of a warp's edges e, e + stride, ...: lanes 0-8 carry the lattice rows, 9-11 the relative position, 12-14
// the reciprocal row lengths, every lane the width of head lane % 8.  Three edges are under way at a time.
struct EdgeStream {
    const float *a, *pos_ij, *tvecs, *rvlen;
    const int64_t *batch, *edges;
    long long E, stride;
    int a_per_edge;
    // current edge
    long long e, i;
    float word, a_own;
    // the next one's values, the one after's crystal, the third's atom
    float word_n, a_n;
    long long i_n, c_n2, i_n2, i_n3;
    int lane;

    __device__ __forceinline__ long long atom(long long at) const { return edges[at < E ? at : E - 1]; }
    __device__ __forceinline__ void fetch(long long at, long long atom_i, long long c, float &w, float &ao) const
    {
        const long long ee = at < E ? at : E - 1;
        const float *src = lane < 9 ? tvecs + 9 * c + lane : lane < 12 ? pos_ij + 3 * ee + (lane - 9)
                           : (lane < 15 && rvlen != nullptr) ? rvlen + 3 * c + (lane - 12) : nullptr;
        w = src != nullptr ? __ldg(src) : 0.f;
        ao = __ldg(a + (a_per_edge ? ee : atom_i) * HEADS + (lane & 7));
    }
    __device__ __forceinline__ void begin(long long first, long long stride_, int lane_)
    {
        e = first; stride = stride_; lane = lane_;
        i = atom(e); i_n = atom(e + stride); i_n2 = atom(e + 2 * stride); i_n3 = atom(e + 3 * stride);
        const long long c0 = batch[i], c1 = batch[i_n];
        c_n2 = batch[i_n2];
        fetch(e, i, c0, word, a_own);
        fetch(e + stride, i_n, c1, word_n, a_n);
    }
    __device__ __forceinline__ void next()
    {
        e += stride;
        i = i_n; i_n = i_n2; i_n2 = i_n3;
        word = word_n; a_own = a_n;
        fetch(e + stride, i_n, c_n2, word_n, a_n);
        c_n2 = batch[i_n2];
        i_n3 = atom(e + 3 * stride);
    }
    __device__ __forceinline__ void unpack(Cell &cell, float &rx, float &ry, float &rz, float (&rvl)[3]) const
    {
        cell.t1x = __shfl_sync(FULL, word, 0); cell.t1y = __shfl_sync(FULL, word, 1); cell.t1z = __shfl_sync(FULL, word, 2);
        cell.t2x = __shfl_sync(FULL, word, 3); cell.t2y = __shfl_sync(FULL, word, 4); cell.t2z = __shfl_sync(FULL, word, 5);
        cell.t3x = __shfl_sync(FULL, word, 6); cell.t3y = __shfl_sync(FULL, word, 7); cell.t3z = __shfl_sync(FULL, word, 8);
        rx = __shfl_sync(FULL, word, 9); ry = __shfl_sync(FULL, word, 10); rz = __shfl_sync(FULL, word, 11);
#pragma unroll
        for (int u = 0; u < 3; ++u) rvl[u] = __shfl_sync(FULL, word, 12 + u);
    }
};

// Digits of translations lane, lane + 32, lane + 64, lane + 96 of the 5 x 5 x 5 box (n3 fastest), as floats.
struct BoxWalk {
    float f1[4], f2[4], f3[4];
    __device__ __forceinline__ void init(int lane)
    {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int t = lane + 32 * b;
            f1[b] = (float)(t / 25 - 2); f2[b] = (float)((t / 5) % 5 - 2); f3[b] = (float)(t % 5 - 2);
        }
    }
};
constexpr int BOX222 = 2 | (2 << 8) | (2 << 16);

__device__ __forceinline__ float term_d2(const Cell &cell, float rx, float ry, float rz, float f1, float f2, float f3)
{
    const float dx = fmaf(cell.t3x, f3, fmaf(cell.t2x, f2, fmaf(cell.t1x, f1, rx)));
    const float dy = fmaf(cell.t3y, f3, fmaf(cell.t2y, f2, fmaf(cell.t1y, f1, ry)));
    const float dz = fmaf(cell.t3z, f3, fmaf(cell.t2z, f2, fmaf(cell.t1z, f1, rz)));
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// Collected terms of a warp: (d2, |n1| | |n2| << 8 | |n3| << 16).
constexpr int EDGE_TERMS = 128;
constexpr int EDGE_TERM_FLOATS = 2 * EDGE_TERMS;
struct EdgeTerms {
    float2 *buf;
    int count, lane;
    __device__ __forceinline__ void add(bool cand, float d2, int key)
    {
        const unsigned mask = __ballot_sync(FULL, cand);
        if (cand) buf[count + __popc(mask & ((1u << lane) - 1u))] = make_float2(d2, __int_as_float(key));
        count += __popc(mask);
    }
    // f(got, d2, key) for every 32 terms; `all`: also the last, incomplete ones (else they stay collected)
    template <class F>
    __device__ __forceinline__ void consume(bool all, F &&f)
    {
        __syncwarp();
        int at = 0;
        for (; at < count && (all || at + 32 <= count); at += 32) {
            const bool got = at + lane < count;
            const float2 en = buf[got ? at + lane : 0];
            f(got, en.x, __float_as_int(en.y));
        }
        const int rest = count - at;
        if (rest > 0) {
            const float2 en = buf[at + (lane < rest ? lane : 0)];
            __syncwarp();
            if (lane < rest) buf[lane] = en;
        }
        count = rest > 0 ? rest : 0;
        __syncwarp();
    }
};

// Walks a box (packed half-widths `uni`) and hands every translation's (valid, d2, f1, f2, f3) to visit; calls full() after
// every 32 of them.
template <class Visit, class Full>
__device__ __forceinline__ void walk_box(const BoxWalk &w5, int uni, const Cell &cell, float rx, float ry, float rz, int lane,
                                         Visit &&visit, Full &&full)
{
    if (uni == BOX222) {
#pragma unroll
        for (int b = 0; b < 4; ++b)
            visit(b < 3 || lane < 29, term_d2(cell, rx, ry, rz, w5.f1[b], w5.f2[b], w5.f3[b]), w5.f1[b], w5.f2[b], w5.f3[b]);
        full();
    } else {
        const int R1 = box_r1(uni), R2 = box_r2(uni), R3 = box_r3(uni);
        const int count = (2 * R1 + 1) * (2 * R2 + 1) * (2 * R3 + 1);
        const float F1 = (float)R1, F2 = (float)R2, F3 = (float)R3;
        TermWalker walk;
        walk.init(R1, R2, R3, (unsigned)lane);
        for (int base = 0; base < count; base += 32) {
            const float f1 = walk.u1 - F1, f2 = walk.u2 - F2, f3 = walk.u3 - F3;
            visit(base + lane < count, term_d2(cell, rx, ry, rz, f1, f2, f3), f1, f2, f3);
            full();
            walk.step();
        }
    }
}

__device__ __forceinline__ int term_key(float f1, float f2, float f3)
{
    return abs(__float2int_rn(f1)) | (abs(__float2int_rn(f2)) << 8) | (abs(__float2int_rn(f3)) << 16);
}
// whether a term's digits are all within the box whose packed half-widths are box (boxor = box | 0x808080): byte-wise
// 128 + R - |n| keeps its top bit exactly when |n| <= R
__device__ __forceinline__ bool term_in_box(int key, int boxor) { return ((boxor - key) & 0x808080) == 0x808080; }

}  // namespace cf
