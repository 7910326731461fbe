// 3x3-block operators of elasticity: the 3 rows of a node have the same columns, which come in
// node triples. Stored as SELL over block rows: slices of B3C block rows, each block row padded
// to its slice's width; a block is 9 values (row-major) and 1 block column; padding blocks are 0
// and point at the block row itself, so that they read x the row reads anyway. Per block 40 bytes
// in FP32 (36 of values, 4 of index) against 72 for the same 9 entries in scalar SELL. The batch
// keeps a block's 9 values together (its threads share a block among right sides); the solver's
// operators keep them in planes (Block3Op).
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <thread>
#include <vector>

#include "hierarchy.hpp"
#include "sell.cuh"

namespace femgpu {

constexpr int B3C = 32;

template <class T>
struct BSell3View {
    int64_t nb;                             // block rows
    const int64_t* __restrict__ slice_ptr;  // in blocks; nslices + 1
    const uint32_t* __restrict__ col;       // block column per block
    const T* __restrict__ val;              // 9 per block
    const uint32_t* __restrict__ row = nullptr;  // the block row of each slot (null: the slot)
};

// The operator of the solver's kernels on the 3x3-block form, its values in planes: value q of
// block k of slice s's row r at val[(9 (slice_ptr[s] / 32 + k) + q) 32 + r], so that the 32 block
// rows of a slice read 9 coalesced runs per block. SPLIT adjacent threads share a block row: each
// takes every SPLIT-th block of it, the 3 sums are joined by shuffles, and row a of the 3 is
// finished by thread a % SPLIT.
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

// Runs f(lo, hi) over [0, n) split among the host threads.
template <class F>
inline void parallel_ranges(int64_t n, F&& f) {
    const int64_t t = std::max<int64_t>(1, std::min<int64_t>(host_threads(), n / 4096));
    if (t == 1) {
        f(0, n);
        return;
    }
    std::vector<std::thread> pool;
    for (int64_t k = 0; k < t; ++k) pool.emplace_back([&, k] { f(n * k / t, n * (k + 1) / t); });
    for (auto& th : pool) th.join();
}

// The 3x3-block SELL form of `a`, if every node's 3 rows have the same columns and the columns
// come in aligned triples; false (and nothing built) otherwise. The block rows are checked and
// filled on all host threads.
template <class T>
inline bool make_bsell3(const HostCsr& a, std::vector<int64_t>* sptr, std::vector<uint32_t>* cols,
                        std::vector<T>* vals) {
    if (a.n % 3 != 0 || a.n / 3 >= 0x7fffffff) return false;
    const int64_t nb = a.n / 3;
    std::vector<int> width(nb);
    std::atomic<bool> ok{true};
    parallel_ranges(nb, [&](int64_t lo, int64_t hi) {
        for (int64_t I = lo; I < hi && ok.load(std::memory_order_relaxed); ++I) {
            const int64_t r0 = 3 * I;
            const int64_t len = a.ptr[r0 + 1] - a.ptr[r0];
            bool good = len % 3 == 0;
            for (int q = 1; q < 3 && good; ++q) {
                if (a.ptr[r0 + q + 1] - a.ptr[r0 + q] != len) good = false;
                for (int64_t k = 0; k < len && good; ++k)
                    if (a.idx[a.ptr[r0 + q] + k] != a.idx[a.ptr[r0] + k]) good = false;
            }
            for (int64_t k = 0; k < len && good; k += 3) {
                const uint32_t c = a.idx[a.ptr[r0] + k];
                if (c % 3 != 0 || a.idx[a.ptr[r0] + k + 1] != c + 1 ||
                    a.idx[a.ptr[r0] + k + 2] != c + 2)
                    good = false;
            }
            if (!good) ok.store(false);
            width[I] = (int)(len / 3);
        }
    });
    if (!ok.load()) return false;
    const int64_t nslices = (nb + B3C - 1) / B3C;
    sptr->assign(nslices + 1, 0);
    for (int64_t sl = 0; sl < nslices; ++sl) {
        int w = 0;
        for (int64_t I = sl * B3C; I < std::min(nb, (sl + 1) * B3C); ++I) w = std::max(w, width[I]);
        (*sptr)[sl + 1] = (*sptr)[sl] + (int64_t)w * B3C;
    }
    cols->assign((*sptr)[nslices], 0);
    vals->assign((size_t)(*sptr)[nslices] * 9, (T)0);
    parallel_ranges(nb, [&](int64_t lo, int64_t hi) {
        for (int64_t I = lo; I < hi; ++I) {
            const int64_t sl = I / B3C, r = I % B3C, base = (*sptr)[sl];
            const int w = (int)(((*sptr)[sl + 1] - base) / B3C);
            for (int k = 0; k < w; ++k) {
                const int64_t blk = base + (int64_t)k * B3C + r;
                if (k < width[I]) {
                    const int64_t e = a.ptr[3 * I] + 3 * k;
                    (*cols)[blk] = a.idx[e] / 3;
                    for (int q = 0; q < 3; ++q)
                        for (int c = 0; c < 3; ++c)
                            (*vals)[(size_t)blk * 9 + 3 * q + c] =
                                (T)a.val[a.ptr[3 * I + q] + 3 * k + c];
                } else {
                    (*cols)[blk] = (uint32_t)I;  // padding: value 0, the block row's own x
                }
            }
        }
    });
    return true;
}

}  // namespace femgpu
