// The multifrontal sparse Cholesky factor on the device (sparse_direct.cuh).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>

#include "rust_format.hpp"
#include "dense_factor.cuh"
#include "sparse_direct.cuh"

namespace femgpu {
namespace {

constexpr double PIVOT = 1e-10;     // cholesky.rs:22
constexpr int SMALL_ROWS = 128;     // fronts factored in shared memory by 1 block
constexpr int CHUNK = 4096;         // entries of an update matrix per extend-add block
constexpr int TH = 256;

// The front of supernode s: m x m, column-major.
struct Fronts {
    const int64_t* first;
    const int64_t* rows_ptr;
    const uint32_t* rows;
    const int64_t* foff;
    double* f;
};

__device__ __forceinline__ int64_t lower_bound(const uint32_t* r, int64_t m, uint32_t v) {
    int64_t lo = 0, hi = m;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (r[mid] < v)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// The entries of A in the lower part of each front (cholesky.rs:60-72), 1 thread per column,
// and each column's diagonal of A.
__global__ void k_assemble_fronts(int64_t n, const int64_t* __restrict__ perm,
                                  const int64_t* __restrict__ iperm,
                                  const int64_t* __restrict__ aptr,
                                  const uint32_t* __restrict__ aidx,
                                  const double* __restrict__ aval,
                                  const int32_t* __restrict__ col2sn, Fronts fr,
                                  double* __restrict__ diag0) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x) {
        const int s = col2sn[j];
        const int64_t r0 = fr.rows_ptr[s], m = fr.rows_ptr[s + 1] - r0;
        const uint32_t* R = fr.rows + r0;
        double* F = fr.f + fr.foff[s] + (j - fr.first[s]) * m;
        const int64_t old = perm[j];
        double d = 0.0;
        for (int64_t e = aptr[old]; e < aptr[old + 1]; ++e) {
            const int64_t i = iperm[aidx[e]];
            if (i == j) d = aval[e];
            if (i >= j) F[lower_bound(R, m, (uint32_t)i)] += aval[e];
        }
        diag0[j] = d;
    }
}

// Extend-add (cholesky.rs:74-86): chunk (child c, part q) adds the lower triangle of a part of
// c's update matrix into its parent's front at the parent's rows.
__global__ void k_extend_add(const int2* __restrict__ chunk, Fronts fr,
                             const int64_t* __restrict__ parent,
                             const uint32_t* __restrict__ relind,
                             const int64_t* __restrict__ relind_off) {
    const int c = chunk[blockIdx.x].x;
    const int64_t q = chunk[blockIdx.x].y;
    const int64_t mc = fr.rows_ptr[c + 1] - fr.rows_ptr[c];
    const int64_t kc = fr.first[c + 1] - fr.first[c];
    const int64_t mu = mc - kc;
    const int64_t p = parent[c];
    const int64_t mp = fr.rows_ptr[p + 1] - fr.rows_ptr[p];
    const double* U = fr.f + fr.foff[c] + kc * mc + kc;
    double* F = fr.f + fr.foff[p];
    const uint32_t* rel = relind + relind_off[c];
    const int64_t end = min(mu * mu, (q + 1) * (int64_t)CHUNK);
    for (int64_t t = q * CHUNK + threadIdx.x; t < end; t += blockDim.x) {
        const int64_t col = t / mu, row = t % mu;
        if (row < col) continue;
        F[rel[row] + (int64_t)rel[col] * mp] += U[row + col * mc];
    }
}

// Partial Cholesky of the first k columns of a front in shared memory (cholesky.rs:173-225):
// each pivot checked against PIVOT times its column's diagonal of A, its column scaled, and the
// rest of the lower triangle updated (right-looking); 1 block per front of at most SMALL_ROWS.
__global__ void __launch_bounds__(TH)
    k_front_small(const int64_t* __restrict__ list, Fronts fr,
                  const double* __restrict__ diag0, unsigned long long* __restrict__ status) {
    extern __shared__ double S[];
    __shared__ int stop;
    const int64_t s = list[blockIdx.x];
    const int64_t j0 = fr.first[s];
    const int m = (int)(fr.rows_ptr[s + 1] - fr.rows_ptr[s]);
    const int k = (int)(fr.first[s + 1] - j0);
    double* F = fr.f + fr.foff[s];
    for (int t = threadIdx.x; t < m * m; t += blockDim.x) S[t] = F[t];
    if (threadIdx.x == 0) stop = 0;
    __syncthreads();
    for (int j = 0; j < k; ++j) {
        if (threadIdx.x == 0) {
            const double d = S[j + j * m];
            if (!(d > PIVOT * fabs(diag0[j0 + j]))) {
                atomicMin(status, (unsigned long long)(j0 + j));
                stop = 1;
            } else {
                S[j + j * m] = sqrt(d);
            }
        }
        __syncthreads();
        if (stop) break;
        const double inv = 1.0 / S[j + j * m];
        for (int r = j + 1 + threadIdx.x; r < m; r += blockDim.x) S[r + j * m] *= inv;
        __syncthreads();
        // The lower triangle of the trailing block, column by column.
        const int w = m - j - 1;
        for (int t = threadIdx.x; t < w * w; t += blockDim.x) {
            const int c = j + 1 + t / w, r = j + 1 + t % w;
            if (r >= c) S[r + c * m] -= S[r + j * m] * S[c + j * m];
        }
        __syncthreads();
    }
    __syncthreads();
    for (int t = threadIdx.x; t < m * m; t += blockDim.x) F[t] = S[t];
}

// ---------------------------------------------------------------- the triangular solves
// Each supernode keeps G = [W; L21 W] (m x k, column-major, leading dimension ld), W = L11^-1:
// with z the supernode's right side (its part of b and its children's updates), the forward
// solve is y1 = W z and z2 -= (L21 W) z, the backward one x1 = G^T [y1; -x2] with x2 the solved
// rows below, stored with the sign in G's lower part (G = [W; -L21 W]). Both are 1 product, so
// every row chunk (or column chunk) of a supernode is its own task with no order between them,
// and a level of the tree is 1 launch over all the level's tasks. A block of 16 warps takes 1
// task with 16 warps, 4 with 4, or 16 with 1, by the supernode's size.
//
// What bounds it: the factor is read once per direction (107 MB for the 36,300-unknown P2 beam:
// 17 us at the copy bandwidth), but a launch per level and direction leaves each level with a
// few microseconds of dependent latency. So each task loads its first entries of G and its
// static indices before it waits for the level before (programmatic dependent launch); after the
// wait only 1 round of loads (the right side) comes before the sums. A block lets the next level
// start as soon as those loads are issued (`early`), so a level's launch and first loads run under
// the levels before it; each still waits for the whole of the level before. The last backward
// level does not: the kernel after it reads x through the read-only path, which must not change
// while that kernel exists. (The trigger at the head of the kernel, before the loads: 541 us where
// this takes 487; at the exit: 556.) The children's updates are
// left in slots grouped by the parent's row, so that the parent reads them as 1 contiguous run.
// Measured on B200: the 50 x 5 x 5 P2 beam's direct solve (2 applications of the factor, 36,300
// unknowns) 3.70 -> 0.80 ms with 22 levels, 0.56 ms with the 11 levels of relaxed supernodes
// (symbolic.cpp), 0.49 ms with the early trigger; the 29,910-unknown coarsest level of a prism
// mesh 1,633 -> 393 -> 199 us, its kernels timed one by one (the early trigger takes 52 us more
// off each iteration of that solve: 22.9 -> 21.0 ms). Before, 1 block took a whole supernode and
// the large ones near the root left the other SMs idle. The error of 1 application against
// extended precision is 1e-12 to 6e-11 on P2 beams of 14,580 to 37,440 unknowns on any form, and its
// residual that of the substitution (k_large_panel).
constexpr int SOLVE_WARPS = 16;
constexpr int SOLVE_TH = 32 * SOLVE_WARPS;
constexpr int ZCAP = 128;  // right side values staged per warp of a task
constexpr int BATCH = 8;   // entries of G in flight per thread
// Columns per warp of a backward task of 1 and of 4 warps (16 warps: 1).
constexpr int COLS_1 = 4, COLS_4 = 2;

__device__ __forceinline__ double slot_sum(double z, const double* slot, uint32_t e0,
                                           uint32_t e1) {
    for (uint32_t e = e0; e < e1; ++e) z += slot[e];
    return z;
}

// A level of the forward solve: task = 32 rows of a supernode, a lane per row, the warps of the
// task splitting its columns.
template <class TB>
__global__ void __launch_bounds__(SOLVE_TH)
    k_sparse_forward(const SolveBlock* __restrict__ blocks, const SolveTask* __restrict__ tasks,
                     const double* __restrict__ G, const uint32_t* __restrict__ slot_ptr,
                     const uint32_t* __restrict__ dst, const int64_t* __restrict__ perm,
                     const TB* b, double* slot, double* yf, int early) {
    __shared__ double zs[SOLVE_WARPS * ZCAP];
    __shared__ double red[SOLVE_TH];
    const SolveBlock B = blocks[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = B.warps, group = warp / nw, wg = warp % nw;
    SolveTask t{};
    if (group < B.count) t = tasks[B.task + group];
    const int row = t.at + lane;
    const bool mine = row < t.m;
    const int kc = min(t.k, t.at + 32);  // W is lower triangular
    const double* col = G + t.g + row;
    double g[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
        const int j = wg + u * nw;
        g[u] = mine && j < kc ? col[(int64_t)j * t.ld] : 0.0;
    }
    const int tid = wg * 32 + lane, gt = nw * 32, cap = ZCAP * nw;
    double* z = zs + group * cap;
    uint32_t e0 = 0, e1 = 0, s0 = 0, s1 = 0, d = 0;
    int64_t pi = 0;
    if (tid < kc) {
        e0 = slot_ptr[t.z + tid];
        e1 = slot_ptr[t.z + tid + 1];
        pi = perm[t.j0 + tid];
    }
    if (wg == 0 && mine && row >= t.k) {
        s0 = slot_ptr[t.z + row];
        s1 = slot_ptr[t.z + row + 1];
        d = dst[t.z + row];
    }
    if (early) pdl_trigger();
    pdl_wait();
    double acc = 0.0;
    // Tasks of fewer than 16 warps have at most `cap` columns: 1 turn for all of the block's.
    const int turns = nw == SOLVE_WARPS ? max(1, (kc + cap - 1) / cap) : 1;
    for (int turn = 0; turn < turns; ++turn) {
        const int c0 = turn * cap, c1 = min(kc, c0 + cap);
        for (int i = c0 + tid; i < c1; i += gt) {
            if (i != tid) {
                e0 = slot_ptr[t.z + i];
                e1 = slot_ptr[t.z + i + 1];
                pi = perm[t.j0 + i];
            }
            z[i - c0] = slot_sum((double)b[pi], slot, e0, e1);
        }
        __syncthreads();
        int j = c0 + wg;
        if (turn == 0) {
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                if (j < c1) acc += g[u] * z[j];
                j += nw;
            }
        }
        for (; j < c1; j += BATCH * nw) {
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int c = j + u * nw;
                g[u] = mine && c < c1 ? col[(int64_t)c * t.ld] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int c = j + u * nw;
                if (c < c1) acc += g[u] * z[c - c0];
            }
        }
        __syncthreads();
    }
    if (nw > 1) {
        red[threadIdx.x] = acc;
        __syncthreads();
        if (wg == 0) {
            acc = 0.0;
            for (int w = 0; w < nw; ++w) acc += red[(warp + w) * 32 + lane];
        }
    }
    if (wg == 0 && mine) {
        if (row < t.k)
            yf[t.j0 + row] = acc;
        else
            slot[d] = slot_sum(0.0, slot, s0, s1) + acc;
    }
}

// A task of the backward solve: up to C columns per warp of a supernode, the lanes along the
// rows, U rows of each column in flight per lane.
template <int C, int U, class TX>
__device__ __forceinline__ void backward_task(const SolveTask& t, int nw, int wg, int lane,
                                              double* v, const double* __restrict__ G,
                                              const uint32_t* __restrict__ rows,
                                              const int64_t* __restrict__ perm,
                                              const double* yf, double* xs, TX* x,
                                              int early) {
    // Column c of the task is column at + c of G; W is lower triangular, so its rows above at
    // are 0.
    const int i0 = t.at & ~3;
    const double* col[C];
    bool on[C];
    double g[U][C], acc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int j = wg + c * nw;
        on[c] = j < t.cols;
        col[c] = G + t.g + (int64_t)(t.at + j) * t.ld;
        acc[c] = 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + 32 * u + lane;
            g[u][c] = on[c] && i < t.m ? col[c][i] : 0.0;
        }
    }
    const int tid = wg * 32 + lane, gt = nw * 32, cap = ZCAP * nw;
    uint32_t r = 0;
    if (i0 + tid < t.m && i0 + tid >= t.k) r = rows[t.z + i0 + tid];
    if (early) pdl_trigger();
    pdl_wait();
    // Tasks of fewer than 16 warps have at most `cap` rows: 1 turn for all of the block's.
    const int turns = nw == SOLVE_WARPS ? max(1, (t.m - i0 + cap - 1) / cap) : 1;
    for (int turn = 0; turn < turns; ++turn) {
        const int c0 = i0 + turn * cap, c1 = min(t.m, c0 + cap);
        for (int i = c0 + tid; i < c1; i += gt) {
            if (i >= t.k && i != i0 + tid) r = rows[t.z + i];
            v[i - c0] = i < t.k ? yf[t.j0 + i] : xs[r];
        }
        __syncthreads();
        for (int i = c0; i < c1; i += 32 * U) {
            if (i != i0) {
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        g[u][c] = on[c] && i + 32 * u + lane < c1 ? col[c][i + 32 * u + lane] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int q = i + 32 * u + lane;
                const double vi = q < c1 ? v[q - c0] : 0.0;
#pragma unroll
                for (int c = 0; c < C; ++c) acc[c] += g[u][c] * vi;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
        double a = acc[c];
#pragma unroll
        for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0 && on[c]) {
            const int64_t j = t.j0 + t.at + wg + c * nw;
            xs[j] = a;
            x[perm[j]] = (TX)a;
        }
    }
}

// A level of the backward solve.
template <class TX>
__global__ void __launch_bounds__(SOLVE_TH)
    k_sparse_backward(const SolveBlock* __restrict__ blocks, const SolveTask* __restrict__ tasks,
                      const double* __restrict__ G, const uint32_t* __restrict__ rows,
                      const int64_t* __restrict__ perm, const double* yf, double* xs, TX* x,
                      int early) {
    __shared__ double vs[SOLVE_WARPS * ZCAP];
    const SolveBlock B = blocks[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = B.warps, group = warp / nw, wg = warp % nw;
    SolveTask t{};
    if (group < B.count) t = tasks[B.task + group];
    double* v = vs + group * ZCAP * nw;
    if (nw == 1)
        backward_task<COLS_1, 2>(t, nw, wg, lane, v, G, rows, perm, yf, xs, x, early);
    else if (nw == 4)
        backward_task<COLS_4, 4>(t, nw, wg, lane, v, G, rows, perm, yf, xs, x, early);
    else
        backward_task<1, 8>(t, nw, wg, lane, v, G, rows, perm, yf, xs, x, early);
}

// ---------------------------------------------------------------- the form of the solves

// G of a supernode of at most 32 columns: 1 block. W by forward substitution, a lane of the
// first warp per column; then a thread per row x of -L21 W, from x L11 = -(its row of L21) by
// substitution in registers.
constexpr int INV_SMALL = 32;
__global__ void __launch_bounds__(128)
    k_small_inverse(const int64_t* __restrict__ list, Fronts fr, const int64_t* __restrict__ goff,
                    const int64_t* __restrict__ gld, double* __restrict__ G) {
    __shared__ double L[INV_SMALL][INV_SMALL + 1], W[INV_SMALL][INV_SMALL + 1];
    const int64_t s = list[blockIdx.x];
    const int64_t m = fr.rows_ptr[s + 1] - fr.rows_ptr[s], ld = gld[s];
    const int k = (int)(fr.first[s + 1] - fr.first[s]);
    const double* F = fr.f + fr.foff[s];
    double* g = G + goff[s];
    for (int e = threadIdx.x; e < INV_SMALL * INV_SMALL; e += blockDim.x) {
        const int i = e % INV_SMALL, j = e / INV_SMALL;
        L[i][j] = i < k && j <= i ? F[i + j * m] : i == j ? 1.0 : 0.0;
        W[i][j] = 0.0;
    }
    __syncthreads();
    if (threadIdx.x < k) {
        const int c = threadIdx.x;
        for (int i = c; i < k; ++i) {
            double v = i == c ? 1.0 : 0.0;
            for (int j = c; j < i; ++j) v -= L[i][j] * W[j][c];
            W[i][c] = v / L[i][i];
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < k * k; e += blockDim.x) g[e % k + (e / k) * ld] = W[e % k][e / k];
    for (int64_t r = k + threadIdx.x; r < m; r += blockDim.x) {
        double x[INV_SMALL];
#pragma unroll
        for (int j = 0; j < INV_SMALL; ++j) x[j] = j < k ? -F[r + j * m] : 0.0;
#pragma unroll
        for (int c = INV_SMALL - 1; c >= 0; --c) {
            x[c] /= L[c][c];
#pragma unroll
            for (int j = 0; j < c; ++j) x[j] -= x[c] * L[c][j];
        }
#pragma unroll
        for (int c = 0; c < INV_SMALL; ++c)
            if (c < k) g[r + c * ld] = x[c];
    }
    for (int64_t r = m + threadIdx.x; r < ld; r += blockDim.x)
        for (int c = 0; c < k; ++c) g[r + c * ld] = 0.0;
}

// The lower triangle of the k x k diagonal block of front F (leading dimension m) into L (leading
// dimension k), zeros above: 1 member of the copy per blockIdx.y.
struct BlockCopy {
    const double* F;
    double* L;
    int64_t m, k;
};

__global__ void k_copy_blocks(const BlockCopy* __restrict__ c) {
    const BlockCopy b = c[blockIdx.y];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < b.k * b.k;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t % b.k, j = t / b.k;
        b.L[t] = i >= j ? b.F[i + j * b.m] : 0.0;
    }
}

// G of the larger supernodes from their W, in 64 x 64 tiles, each sum over the columns in order:
//   0: G = [W; -L21 W];
//   1: E = L21 + G2 L11, what that lower part X = -G2 leaves of X L11 = L21, in place of L21;
//   2: G2 -= E W.
// The step of refinement brings X back to a substitution's accuracy. With L21 W as it is rounded, an
// application of the factor left 1.1 times the residual on P2 beams (2e-18 of the terms' size), 1.5
// times with a Poisson ratio of 0.4999; the setup takes 6 of 330 ms more for 36,300 unknowns.
struct GTile {
    double* F;
    const double* W;
    double* g;
    int64_t m, k, ld;
    int r0, c0;
};

template <int STEP>
__global__ void __launch_bounds__(TH) k_large_panel(const GTile* __restrict__ tiles) {
    constexpr int KT = 16;
    __shared__ double A[KT][64], Bs[KT][64 + 1];
    const GTile t = tiles[blockIdx.x];
    if (STEP > 0 && t.r0 + 64 <= t.k) return;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    double acc[4][4] = {};
    // W and L11 are lower triangular: column c starts at row c.
    for (int64_t k0 = t.c0; k0 < t.k; k0 += KT) {
        for (int e = threadIdx.x; e < KT * 64; e += TH) {
            const int r = e % 64, q = e / 64;
            const int64_t i = t.r0 + r, j = k0 + q;
            const bool in = j < t.k && i < t.m;
            // L21 (or E), or the identity where the tile's rows are W's own; or G2.
            if (STEP == 1)
                A[q][r] = in && i >= t.k ? -t.g[i + j * t.ld] : 0.0;
            else
                A[q][r] = !in ? 0.0 : i >= t.k ? t.F[i + j * t.m] : i == j ? -1.0 : 0.0;
        }
        for (int e = threadIdx.x; e < KT * 64; e += TH) {
            const int q = e % KT, c = e / KT;
            const int64_t j = k0 + q, col = t.c0 + c;
            const bool in = j < t.k && col < t.k;
            if (STEP == 1)
                Bs[q][c] = in && j >= col ? t.F[j + col * t.m] : 0.0;
            else
                Bs[q][c] = in ? t.W[j + col * t.k] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < KT; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] -= A[q][tx + 16 * i] * Bs[q][ty + 16 * j];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t r = t.r0 + tx + 16 * i, c = t.c0 + ty + 16 * j;
            if (STEP == 0 && r < t.ld && c < t.k) t.g[r + c * t.ld] = acc[i][j];
            if (STEP == 1 && r >= t.k && r < t.m && c < t.k) t.F[r + c * t.m] += acc[i][j];
            if (STEP == 2 && r >= t.k && r < t.m && c < t.k) t.g[r + c * t.ld] += acc[i][j];
        }
}

}  // namespace

void SparseFactor::factor(const HostCsr& a, const double* xyz, cudaStream_t s) {
    n_ = a.n;
    // The reference's fill-reducing order (order.rs) and the analysis in it.
    Supernodal S = analyse_factor(a, nested_dissection(a, xyz));
    ns_ = S.ns;
    entries_ = S.entries;
    flops_ = S.flops;
    m_.resize(ns_);
    k_.resize(ns_);
    std::vector<int64_t> foff(ns_);
    size_t fv = 0;
    for (int64_t t = 0; t < ns_; ++t) {
        m_[t] = S.rows_ptr[t + 1] - S.rows_ptr[t];
        k_[t] = S.first[t + 1] - S.first[t];
        foff[t] = (int64_t)fv;
        fv += (size_t)(m_[t] * m_[t]);
    }
    front_values_ = fv;
    if (fv > ((size_t)96 << 30) / 8)
        throw Failure(FEMGPU_ERR_TOO_LARGE,
                      "the frontal matrices of the sparse factor need more than 96 GiB");
    // Children (increasing), relative indices of each child's update rows in its parent.
    std::vector<int64_t> cptr(ns_ + 1, 0), clist;
    for (int64_t t = 0; t < ns_; ++t)
        if (S.parent[t] >= 0) cptr[S.parent[t] + 1] += 1;
    for (int64_t t = 0; t < ns_; ++t) cptr[t + 1] += cptr[t];
    clist.resize(cptr[ns_]);
    std::vector<int64_t> fill(cptr.begin(), cptr.end() - 1);
    for (int64_t t = 0; t < ns_; ++t)
        if (S.parent[t] >= 0) clist[fill[S.parent[t]]++] = t;
    std::vector<int64_t> roff(ns_, 0);
    std::vector<uint32_t> rel;
    for (int64_t c = 0; c < ns_; ++c) {
        roff[c] = (int64_t)rel.size();
        const int64_t p = S.parent[c];
        if (p < 0) continue;
        const uint32_t* Rp = S.rows.data() + S.rows_ptr[p];
        for (int64_t t = S.rows_ptr[c] + k_[c]; t < S.rows_ptr[c + 1]; ++t)
            rel.push_back((uint32_t)(std::lower_bound(Rp, Rp + m_[p], S.rows[t]) - Rp));
    }
    // The level schedule.
    height_ = 0;
    for (int h : S.height) height_ = std::max<int64_t>(height_, h);
    std::vector<std::vector<int64_t>> small(height_ + 1), large(height_ + 1);
    levels_.assign(height_ + 1, {});
    large_fronts_ = 0;
    for (int64_t t = 0; t < ns_; ++t) {
        (m_[t] <= SMALL_ROWS ? small : large)[S.height[t]].push_back(t);
        large_fronts_ += m_[t] > SMALL_ROWS;
        levels_[S.height[t]].push_back(t);
    }
    std::vector<int64_t> sl, small_at(1, 0);
    for (int64_t h = 0; h <= height_; ++h) {
        sl.insert(sl.end(), small[h].begin(), small[h].end());
        small_at.push_back((int64_t)sl.size());
    }
    // The slots of the forward solve: the update that row r of a supernode gets from each child,
    // a row's slots together and in the children's order.
    host_zoff_.assign(S.rows_ptr.begin(), S.rows_ptr.end() - 1);
    const size_t nrows = S.rows.size();
    if (nrows >= (size_t)UINT32_MAX) throw Failure(FEMGPU_ERR_TOO_LARGE, "too many factor rows");
    std::vector<uint32_t> slot_ptr(nrows + 1, 0), dst(nrows, 0);
    for (int64_t c = 0; c < ns_; ++c)
        if (S.parent[c] >= 0)
            for (int64_t t = 0; t < m_[c] - k_[c]; ++t)
                slot_ptr[S.rows_ptr[S.parent[c]] + rel[roff[c] + t] + 1] += 1;
    for (size_t t = 0; t < nrows; ++t) slot_ptr[t + 1] += slot_ptr[t];
    std::vector<uint32_t> next(slot_ptr.begin(), slot_ptr.end() - 1);
    for (int64_t c = 0; c < ns_; ++c)
        if (S.parent[c] >= 0)
            for (int64_t t = 0; t < m_[c] - k_[c]; ++t)
                dst[S.rows_ptr[c] + k_[c] + t] =
                    next[S.rows_ptr[S.parent[c]] + rel[roff[c] + t]]++;
    // Extend-add chunks per (height of the parent, rank of the child).
    std::vector<int2> ch;
    struct Chunks {
        int64_t height, at, count;  // into ch
    };
    std::vector<Chunks> chunks;
    for (int64_t h = 1; h <= height_; ++h) {
        int maxrank = -1;
        for (int64_t p : levels_[h]) maxrank = std::max<int>(maxrank, (int)(cptr[p + 1] - cptr[p]) - 1);
        for (int r = 0; r <= maxrank; ++r) {
            Chunks c{h, (int64_t)ch.size(), 0};
            for (int64_t p : levels_[h]) {
                if (cptr[p + 1] - cptr[p] <= r) continue;
                const int64_t cc = clist[cptr[p] + r];
                const int64_t mu = m_[cc] - k_[cc];
                const int64_t parts = (mu * mu + CHUNK - 1) / CHUNK;
                for (int64_t q = 0; q < parts; ++q) ch.push_back(int2{(int)cc, (int)q});
            }
            c.count = (int64_t)ch.size() - c.at;
            if (c.count) chunks.push_back(c);
        }
    }
    if (ns_ >= INT_MAX) throw Failure(FEMGPU_ERR_TOO_LARGE, "too many supernodes");
    // Device arrays.
    std::vector<int32_t> col2sn(n_);
    for (int64_t t = 0; t < ns_; ++t)
        for (int64_t j = S.first[t]; j < S.first[t + 1]; ++j) col2sn[j] = (int32_t)t;
    perm_.upload(S.perm.data(), n_, s);
    DevBuf<int64_t> iperm;
    iperm.upload(S.iperm.data(), n_, s);
    first_.upload(S.first.data(), ns_ + 1, s);
    rows_ptr_.upload(S.rows_ptr.data(), ns_ + 1, s);
    rows_.upload(S.rows.data(), S.rows.size(), s);
    foff_.upload(foff.data(), ns_, s);
    host_foff_ = foff;
    host_first_ = S.first;
    slot_ptr_.upload(slot_ptr.data(), nrows + 1, s);
    dst_.upload(dst.data(), nrows, s);
    slot_.alloc(std::max<size_t>(1, slot_ptr[nrows]));
    DevBuf<uint32_t> relind;
    DevBuf<int64_t> relind_off, small_list, parent;
    DevBuf<int2> chunk;
    relind.upload(rel.data(), rel.size(), s);
    relind_off.upload(roff.data(), ns_, s);
    small_list.upload(sl.data(), sl.size(), s);
    chunk.upload(ch.data(), ch.size(), s);
    parent.upload(S.parent.data(), ns_, s);
    DevBuf<int32_t> dcol2sn;
    dcol2sn.upload(col2sn.data(), n_, s);
    fronts_.alloc(fv);
    FG_CUDA(cudaMemsetAsync(fronts_.p, 0, fv * sizeof(double), s));
    y_.alloc(n_);
    xs_.alloc(n_);
    DevBuf<int64_t> aptr;
    DevBuf<uint32_t> aidx;
    DevBuf<double> aval, diag0(n_);
    aptr.upload(a.ptr.data(), n_ + 1, s);
    aidx.upload(a.idx.data(), a.nnz(), s);
    aval.upload(a.val.data(), a.nnz(), s);
    DevBuf<unsigned long long> status(1);
    FG_CUDA(cudaMemsetAsync(status.p, 0xff, sizeof(unsigned long long), s));
    const Fronts fr{first_.p, rows_ptr_.p, rows_.p, foff_.p, fronts_.p};
    k_assemble_fronts<<<blocks_for(n_, TH), TH, 0, s>>>(n_, perm_.p, iperm.p, aptr.p, aidx.p,
                                                       aval.p, dcol2sn.p, fr, diag0.p);
    FG_CHECK_LAUNCH();
    const size_t smem = (size_t)SMALL_ROWS * SMALL_ROWS * sizeof(double);
    FG_CUDA(cudaFuncSetAttribute(k_front_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    size_t ci = 0;
    for (int64_t h = 0; h <= height_; ++h) {
        for (; ci < chunks.size() && chunks[ci].height == h; ++ci)
            k_extend_add<<<(unsigned)chunks[ci].count, TH, 0, s>>>(
                chunk.p + chunks[ci].at, fr, parent.p, relind.p, relind_off.p);
        const int64_t ns_small = small_at[h + 1] - small_at[h];
        if (ns_small > 0) {
            int mmax = 0;
            for (int64_t t : small[h]) mmax = std::max<int>(mmax, (int)m_[t]);
            k_front_small<<<(unsigned)ns_small, TH, (size_t)mmax * mmax * sizeof(double), s>>>(
                small_list.p + small_at[h], fr, diag0.p, status.p);
        }
        for (int64_t t : large[h])
            dense_partial_cholesky(fronts_.p + foff[t], m_[t], k_[t], diag0.p + S.first[t],
                                   S.first[t], status.p, s);
        FG_CHECK_LAUNCH();
    }
    unsigned long long bad = fetch(status.p, s);
    if (bad != ~0ull) {
        const int64_t j = (int64_t)bad;
        const double d = fetch(diag0.p + j, s);
        char buf[320];
        std::snprintf(buf, sizeof buf,
                      "the matrix is not positive definite: the pivot of column %lld is 0 or less "
                      "to the precision of the arithmetic (its diagonal is %s)",
                      (long long)S.perm[j], rust_exp_shortest(d).c_str());
        throw Failure(FEMGPU_ERR_NOT_SPD, buf);
    }
    pack(s);
}

// The supernodes' G panels from the fronts, which are then freed.
void SparseFactor::pack(cudaStream_t s) {
    std::vector<int64_t> goff(ns_), gld(ns_);
    int64_t total = 0;
    std::vector<int64_t> small, large;
    for (int64_t t = 0; t < ns_; ++t) {
        gld[t] = (m_[t] + 3) & ~(int64_t)3;  // columns start on 32-byte sectors
        goff[t] = total;
        total += gld[t] * k_[t];
        (k_[t] <= INV_SMALL ? small : large).push_back(t);
    }
    g_.alloc(std::max<int64_t>(1, total));
    DevBuf<int64_t> dgoff, dgld, dsmall;
    dgoff.upload(goff.data(), ns_, s);
    dgld.upload(gld.data(), ns_, s);
    const Fronts fr{first_.p, rows_ptr_.p, rows_.p, foff_.p, fronts_.p};
    if (!small.empty()) {
        dsmall.upload(small.data(), small.size(), s);
        k_small_inverse<<<(unsigned)small.size(), 128, 0, s>>>(dsmall.p, fr, dgoff.p, dgld.p,
                                                               g_.p);
        FG_CHECK_LAUNCH();
    }
    // The larger ones' W by the batched triangular inverse, a bounded number at a time.
    constexpr size_t AT_ONCE = 4096;
    constexpr int64_t VALUES_AT_ONCE = (int64_t)1 << 27;
    for (size_t at = 0, end; at < large.size(); at = end) {
        int64_t kk = 0, kmax = 0;
        for (end = at; end < large.size() && end - at < AT_ONCE; ++end) {
            const int64_t k = k_[large[end]];
            if (end > at && kk + k * k > VALUES_AT_ONCE) break;
            kk += k * k;
            kmax = std::max(kmax, k);
        }
        DevBuf<double> lc(kk), wc(kk);
        std::vector<BlockCopy> bc;
        std::vector<GTile> tiles;
        std::vector<int64_t> n;
        std::vector<double*> ls, ws;
        int64_t off = 0;
        for (size_t e = at; e < end; ++e) {
            const int64_t t = large[e];
            double* F = fronts_.p + host_foff_[t];
            bc.push_back({F, lc.p + off, m_[t], k_[t]});
            n.push_back(k_[t]);
            ls.push_back(lc.p + off);
            ws.push_back(wc.p + off);
            for (int64_t r0 = 0; r0 < gld[t]; r0 += 64)
                for (int64_t c0 = 0; c0 < k_[t]; c0 += 64)
                    tiles.push_back(GTile{F, wc.p + off, g_.p + goff[t], m_[t], k_[t], gld[t],
                                          (int)r0, (int)c0});
            off += k_[t] * k_[t];
        }
        DevBuf<BlockCopy> dbc;
        dbc.upload(bc.data(), bc.size(), s);
        k_copy_blocks<<<dim3((unsigned)blocks_for(kmax * kmax, TH, 256), (unsigned)bc.size()), TH,
                        0, s>>>(dbc.p);
        FG_CHECK_LAUNCH();
        DenseBatchWork w;
        triangular_inverse_batch(n, ls, ws, &w, s);
        DevBuf<GTile> dt;
        dt.upload(tiles.data(), tiles.size(), s);
        k_large_panel<0><<<(unsigned)tiles.size(), TH, 0, s>>>(dt.p);
        k_large_panel<1><<<(unsigned)tiles.size(), TH, 0, s>>>(dt.p);
        k_large_panel<2><<<(unsigned)tiles.size(), TH, 0, s>>>(dt.p);
        FG_CHECK_LAUNCH();
        FG_CUDA(cudaStreamSynchronize(s));
    }
    // The tasks of each level.
    std::vector<SolveBlock> fb, bb;
    std::vector<SolveTask> ft, bt;
    forward_at_.assign(1, 0);
    backward_at_.assign(1, 0);
    // Tasks of 16, 4 and 1 warps go to blocks of their own kind; the long ones first.
    auto flush = [&](std::vector<SolveTask> (&kind)[3], std::vector<SolveTask>& tasks,
                     std::vector<SolveBlock>& blocks) {
        for (int q = 0; q < 3; ++q) {
            const int warps = q == 0 ? 16 : q == 1 ? 4 : 1, per = SOLVE_WARPS / warps;
            for (size_t e = 0; e < kind[q].size(); e += per)
                blocks.push_back(SolveBlock{(int)(tasks.size() + e),
                                            (int)std::min<size_t>(per, kind[q].size() - e), warps});
            tasks.insert(tasks.end(), kind[q].begin(), kind[q].end());
        }
    };
    for (int64_t h = 0; h <= height_; ++h) {
        std::vector<SolveTask> fk[3], bk[3];
        for (int64_t t : levels_[h]) {
            SolveTask q{};
            q.g = goff[t];
            q.z = host_zoff_[t];
            q.j0 = host_first_[t];
            q.ld = (int)gld[t];
            q.m = (int)m_[t];
            q.k = (int)k_[t];
            // Forward: at most 32 entries of G per thread up to 128 columns (a warp alone up to
            // 32, 4 warps up to 128), 16 warps above.
            const int fq = k_[t] <= 32 ? 2 : k_[t] <= 128 ? 1 : 0;
            for (int64_t r = 0; r < m_[t]; r += 32) {
                q.at = (int)r;
                fk[fq].push_back(q);
            }
            // Backward: 1 warp takes 4 columns of up to 128 rows, 4 warps 2 columns each of up
            // to 512, 16 warps 1 column each above: 16 to 32 entries of G per thread.
            const int bq = m_[t] <= ZCAP - 4 ? 2 : m_[t] <= 4 * ZCAP - 4 ? 1 : 0;
            const int step = bq == 2 ? COLS_1 : bq == 1 ? 4 * COLS_4 : 16;
            for (int64_t c = 0; c < k_[t]; c += step) {
                q.at = (int)c;
                q.cols = (int)std::min<int64_t>(step, k_[t] - c);
                bk[bq].push_back(q);
            }
        }
        flush(fk, ft, fb);
        flush(bk, bt, bb);
        forward_at_.push_back((int64_t)fb.size());
        backward_at_.push_back((int64_t)bb.size());
    }
    forward_blocks_.upload(fb.data(), fb.size(), s);
    backward_blocks_.upload(bb.data(), bb.size(), s);
    forward_tasks_.upload(ft.data(), ft.size(), s);
    backward_tasks_.upload(bt.data(), bt.size(), s);
    FG_CUDA(cudaStreamSynchronize(s));
    fronts_.release();
}

template <class TB, class TX>
void SparseFactor::solve(const TB* b, TX* x, bool pdl, cudaStream_t s) {
    for (int64_t h = 0; h <= height_; ++h)
        launch(pdl, k_sparse_forward<TB>, (int)(forward_at_[h + 1] - forward_at_[h]), SOLVE_TH, s,
               forward_blocks_.p + forward_at_[h], forward_tasks_.p, g_.p, slot_ptr_.p, dst_.p,
               perm_.p, b, slot_.p, y_.p, 1);
    for (int64_t h = height_; h >= 0; --h)
        launch(pdl, k_sparse_backward<TX>, (int)(backward_at_[h + 1] - backward_at_[h]), SOLVE_TH,
               s, backward_blocks_.p + backward_at_[h], backward_tasks_.p, g_.p, rows_.p, perm_.p,
               y_.p, xs_.p, x, h > 0 ? 1 : 0);
}
template void SparseFactor::solve<double, double>(const double*, double*, bool, cudaStream_t);
template void SparseFactor::solve<float, float>(const float*, float*, bool, cudaStream_t);

size_t SparseFactor::solve_launches() const {
    return 2 * (size_t)(height_ + 1);
}

size_t SparseFactor::bytes() const {
    return fronts_.bytes() + g_.bytes() + y_.bytes() + xs_.bytes() + slot_.bytes() +
           slot_ptr_.bytes() + dst_.bytes() + perm_.bytes() + first_.bytes() +
           rows_ptr_.bytes() + rows_.bytes() + foff_.bytes() + forward_blocks_.bytes() +
           backward_blocks_.bytes() + forward_tasks_.bytes() + backward_tasks_.bytes();
}

std::string SparseFactor::describe() const {
    char buf[256];
    int64_t mmax = 0;
    for (int64_t m : m_) mmax = std::max(mmax, m);
    std::snprintf(buf, sizeof buf,
                  "sparse multifrontal factor: %lld supernodes, %lld levels, %lld fronts above %d "
                  "rows (largest %lld), L entries %llu, flops %.3g, front values %zu\n",
                  (long long)ns_, (long long)height_ + 1, (long long)large_fronts_, SMALL_ROWS,
                  (long long)mmax, (unsigned long long)entries_, flops_, front_values_);
    return buf;
}

}  // namespace femgpu
