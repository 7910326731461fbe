// 3x3-block operators of elasticity: the 3 rows of a node have the same columns, which come in
// node triples. Stored as SELL over block rows: slices of B3C block rows, each block row padded
// to its slice's width; a block is 9 values (row-major) and 1 block column; padding blocks are 0
// and point at the block row itself, so that they read x the row reads anyway. The values are in
// planes: value q of block k of slice s's row r at val[(9 (slice_ptr[s] / 32 + k) + q) 32 + r], so
// that the 32 block rows of a slice read 9 coalesced runs per block. Per block 40 bytes
// in FP32 (36 of values, 4 of index) against 72 for the same 9 entries in scalar SELL.
#pragma once
#include <cstdint>

#include "sell.cuh"

namespace femgpu {

constexpr int B3C = 32;

template <class T>
struct BSell3View {
    int64_t nb;                             // block rows
    const int64_t* __restrict__ slice_ptr;  // in blocks; nslices + 1
    const uint32_t* __restrict__ col;       // block column per block
    const T* __restrict__ val;              // 9 planes per 32 blocks
    const uint32_t* __restrict__ row = nullptr;  // the block row of each slot (null: the slot)
};

// The operator of the solver's kernels on the 3x3-block form. SPLIT adjacent threads share a block
// row: each takes every SPLIT-th block of it, the 3 sums are joined by shuffles, and row a of the 3
// is finished by thread a % SPLIT.
//
// `head` loads a thread's first AHEAD blocks; a kernel calls it before it waits for the kernel
// before it, since the operator itself does not change. `apply` keeps one batch ahead: the next
// blocks' values and columns are on their way while x is gathered for the current ones.
//
// A slice stores its longest row's width for all 32 rows, so the block rows of a window are sorted
// by width where that saves blocks (`row` maps a slot to its block row): 13 % of the blocks of a
// P2 box mesh were padding and 29 % of a P2 prism mesh's, 1 % and 3 % after.
//
// What bounds it: the values and columns, each read once (HBM). Measured on B200 against 1 row per
// thread with a block's 9 values together (3 strided loads per thread and block, and each of the
// 3 threads loading column and x): finest smoothing step in FP32 and FP64 product q = A p of
//   box cells 256 x 32 x 32 (278,784 block rows):   62.8 -> 54 us, 103 -> 87 us
//   P2 beam 200 x 20 x 20 (672,400):                168 -> 140 us, 268 -> 225 us
//   P2 prism plate (219,209):                         72 -> 58 us, 110 -> 78 us
// and an iteration of their mixed solves 500 -> 437, 1,174 -> 1,016 and 788 -> 682 us.
template <class T, int SPLIT>
struct Block3Op {
    static constexpr int ROWS = 3;
    static constexpr int AHEAD = sizeof(T) == 4 && SPLIT == 1 ? 3 : 2;
    BSell3View<T> v;
    int n;  // rows = 3 nb
    struct Batch {
        uint32_t col[AHEAD];
        T a[AHEAD][9];
    };
    struct Head {
        int64_t base;  // the slice's first block over 32
        int width;     // 0 past the last slot
        int I;         // the block row
        Batch first;
    };
    __host__ __device__ __forceinline__ int64_t threads() const {
        return (v.nb + B3C - 1) / B3C * B3C * SPLIT;
    }
    // The blocks k, k + SPLIT, ... of slot `slot`.
    __device__ __forceinline__ void load(const Head& h, int slot, int k, Batch* out) const {
        const int r = slot % B3C;
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const bool in = k + u * SPLIT < h.width;
            const int64_t at = (h.base + k + u * SPLIT) * B3C + r;
            const T* val = v.val + (h.base + k + u * SPLIT) * (9 * B3C) + r;
            out->col[u] = in ? __ldg(v.col + at) : (uint32_t)h.I;
#pragma unroll
            for (int q = 0; q < 9; ++q) out->a[u][q] = in ? __ldg(val + q * B3C) : (T)0;
        }
    }
    __device__ __forceinline__ Head head(int t) const {
        Head h;
        const int slot = t / SPLIT;
        h.base = 0;
        h.width = 0;
        h.I = 0;
        if (slot < v.nb) {
            const int64_t b = __ldg(v.slice_ptr + slot / B3C);
            const int64_t e = __ldg(v.slice_ptr + slot / B3C + 1);
            h.base = b / B3C;
            h.width = (int)((e - b) / B3C);
            h.I = v.row ? (int)__ldg(v.row + slot) : slot;
        }
        load(h, slot, t % SPLIT, &h.first);
        return h;
    }
    // f(row, its sum) for the rows that this thread finishes. Every lane of the warp calls it.
    template <class TA, class TX, class F>
    __device__ __forceinline__ void apply(const Head& h, int t, const TX* __restrict__ x,
                                          F&& f) const {
        const int slot = t / SPLIT;
        TA s[3] = {0, 0, 0};
        Batch cur = h.first;
        for (int k = t % SPLIT; k < h.width; k += AHEAD * SPLIT) {
            TX xv[AHEAD][3];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c) xv[u][c] = __ldg(x + 3 * (int64_t)cur.col[u] + c);
            Batch next;
            load(h, slot, k + AHEAD * SPLIT, &next);
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int a = 0; a < 3; ++a) s[a] += (TA)cur.a[u][3 * a + c] * (TA)xv[u][c];
            cur = next;
        }
#pragma unroll
        for (int o = 1; o < SPLIT; o *= 2)
#pragma unroll
            for (int a = 0; a < 3; ++a) s[a] += __shfl_xor_sync(0xffffffffu, s[a], o);
        if (slot >= v.nb) return;
#pragma unroll
        for (int a = 0; a < 3; ++a)
            if (a % SPLIT == t % SPLIT) f(3 * h.I + a, s[a]);
    }
};

}  // namespace femgpu
