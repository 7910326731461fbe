// The inverse of a dense SPD matrix (spd_inverse.cuh).
#include "spd_inverse.cuh"

namespace femgpu {
namespace {

constexpr double PIVOT = 1e-10;  // cholesky.rs:22
constexpr int NB = SPD_BLOCK;
constexpr int TH = 256;
constexpr int KC = 16;       // inner terms staged at a time
constexpr int STAGES = 3;
constexpr int LDT = NB + 4;  // 4 mod 16: the 16 fragments of a half warp fall in 16 banks
constexpr int PR = 32;       // rows of a panel piece
constexpr int LDP = PR + 4;

constexpr size_t TILE_SMEM = (size_t)STAGES * 2 * KC * LDT * sizeof(double);
constexpr size_t DIAG_SMEM = (size_t)NB * LDT * sizeof(double);
constexpr size_t STEP_SMEM = TILE_SMEM > DIAG_SMEM ? TILE_SMEM : DIAG_SMEM;
constexpr size_t PANEL_SMEM = (2 * (size_t)NB * LDP + (size_t)NB * LDT) * sizeof(double);

// D += A B on the FP64 tensor cores: A 16 x 8, B 8 x 8, D 16 x 8. Lane l with g = l / 4 and
// q = l % 4 holds A[g][q], A[g + 8][q], A[g][q + 4], A[g + 8][q + 4], B[q][g], B[q + 4][g] and
// D[g][2q], D[g][2q + 1], D[g + 8][2q], D[g + 8][2q + 1].
__device__ __forceinline__ void dmma16(double (&d)[4], const double (&a)[4], double b0,
                                       double b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

__device__ __forceinline__ void copy16(double* to, const double* from) {
    const unsigned t = (unsigned)__cvta_generic_to_shared(to);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(t), "l"(from) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// acc += the 128 x 128 product sum_k A[i + k ld] B[j + k ld] over k < kn (a multiple of KC).
// Warp w takes rows 64 (w % 2) and columns 32 (w / 2), in 4 x 4 products of 16 x 8.
__device__ __forceinline__ void tile_product(const double* __restrict__ A,
                                             const double* __restrict__ B, int64_t ld, int kn,
                                             double* sm, double (&acc)[4][4][4]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int r0 = 64 * (warp & 1) + g, c0 = 32 * (warp >> 1) + g;
    const int turns = kn / KC;
    auto fetch = [&](int t) {
        if (t < turns) {
            double* as = sm + (t % STAGES) * 2 * KC * LDT;
            double* bs = as + KC * LDT;
            for (int e = threadIdx.x; e < KC * NB / 2; e += TH) {
                const int r = 2 * (e % (NB / 2)), k = e / (NB / 2);
                copy16(as + k * LDT + r, A + r + (int64_t)(t * KC + k) * ld);
                copy16(bs + k * LDT + r, B + r + (int64_t)(t * KC + k) * ld);
            }
        }
        copy_commit();
    };
    __syncthreads();
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) fetch(t);
    for (int t = 0; t < turns; ++t) {
        copy_wait<STAGES - 2>();
        __syncthreads();
        fetch(t + STAGES - 1);
        const double* as = sm + (t % STAGES) * 2 * KC * LDT;
        const double* bs = as + KC * LDT;
#pragma unroll
        for (int kk = 0; kk < KC; kk += 8) {
            double a[4][4], b[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[i][0] = as[(kk + q) * LDT + r0 + 16 * i];
                a[i][1] = as[(kk + q) * LDT + r0 + 16 * i + 8];
                a[i][2] = as[(kk + q + 4) * LDT + r0 + 16 * i];
                a[i][3] = as[(kk + q + 4) * LDT + r0 + 16 * i + 8];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                b[j][0] = bs[(kk + q) * LDT + c0 + 8 * j];
                b[j][1] = bs[(kk + q + 4) * LDT + c0 + 8 * j];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma16(acc[i][j], a[i], b[j][0], b[j][1]);
        }
    }
    copy_wait<0>();
    __syncthreads();
}

// f(row, column, acc's value) for each of the thread's 64 values of a tile.
template <class F>
__device__ __forceinline__ void each_value(double (&acc)[4][4][4], F&& f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = 64 * (warp & 1) + (lane >> 2), c0 = 32 * (warp >> 1) + 2 * (lane & 3);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 4; ++h)
                f(r0 + 16 * i + 8 * (h >> 1), c0 + 8 * j + (h & 1), acc[i][j][h]);
}

// C -= acc, 32 values of C in flight per thread.
__device__ __forceinline__ void take_off(const double (&acc)[4][4][4], double* C, int64_t ld) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* c0 = C + 64 * (warp & 1) + (lane >> 2) +
                 (int64_t)(32 * (warp >> 1) + 2 * (lane & 3)) * ld;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        double v[2][4][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    v[i][j][h] = c0[32 * half + 16 * i + 8 * (h >> 1) +
                                    (int64_t)(8 * j + (h & 1)) * ld];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    c0[32 * half + 16 * i + 8 * (h >> 1) + (int64_t)(8 * j + (h & 1)) * ld] =
                        v[i][j][h] - acc[2 * half + i][j][h];
    }
}

// The diagonal block in D (row i at i LDT, its lower triangle): its Cholesky factor in place and
// the inverse W of that factor, W[i][j] at D[j LDT + i + 1] (above the diagonal); `pair` gets
// D. By 32 columns: the first warp factors
// the 32 x 32 block with a lane per row, the rows below are solved a thread each, the rest is
// updated by tensor core products; then W by block rows.
__device__ void diagonal_block(double* D, const double* __restrict__ diag, int64_t col0, int live,
                               double* __restrict__ pair,
                               unsigned long long* __restrict__ status) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    __syncthreads();
    for (int p = 0; p < NB; p += 32) {
        if (warp == 0) {
            double a[32];
            const double lim = p + lane < live ? PIVOT * fabs(diag[col0 + p + lane]) : 0.0;
#pragma unroll
            for (int j = 0; j < 32; ++j) a[j] = j <= lane ? D[(p + lane) * LDT + p + j] : 0.0;
            bool bad = false;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const double d = __shfl_sync(0xffffffffu, a[j], j);
                if (lane == j && !(d > lim)) bad = true;
                // 1 special function per pivot, on the block's serial chain.
                const double inv = rsqrt(d);
                a[j] = (lane == j ? d : a[j]) * inv;
                if (lane == j) D[(p + j) * LDT + p + j + 1] = inv;
#pragma unroll
                for (int c = 1; c < 32; ++c)
                    if (c > j) {
                        const double l = __shfl_sync(0xffffffffu, a[j], c);
                        if (lane >= c) a[c] -= a[j] * l;
                    }
            }
            if (bad && p + lane < live) atomicMin(status, (unsigned long long)(col0 + p + lane));
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (j <= lane) D[(p + lane) * LDT + p + j] = a[j];
        }
        __syncthreads();
        const int below = NB - p - 32;
        if (tid < below) {
            double x[32];
            double* row = D + (p + 32 + tid) * LDT + p;
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = row[j];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                x[j] *= D[(p + j) * LDT + p + j + 1];
#pragma unroll
                for (int c = 1; c < 32; ++c)
                    if (c > j) x[c] -= x[j] * D[(p + c) * LDT + p + j];
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) row[j] = x[j];
        }
        __syncthreads();
        // The lower tiles, 16 x 8, of the rest minus the products of the 32 columns.
        const int across = below / 8;
        for (int e = warp; e < below / 16 * across; e += TH / 32) {
            const int i0 = p + 32 + 16 * (e / across), j0 = p + 32 + 8 * (e % across);
            if (j0 >= i0 + 16) continue;
            double s[4] = {};
#pragma unroll
            for (int k = p; k < p + 32; k += 8) {
                const double u[4] = {D[(i0 + g) * LDT + k + q], D[(i0 + g + 8) * LDT + k + q],
                                     D[(i0 + g) * LDT + k + q + 4],
                                     D[(i0 + g + 8) * LDT + k + q + 4]};
                dmma16(s, u, D[(j0 + g) * LDT + k + q], D[(j0 + g) * LDT + k + q + 4]);
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int i = i0 + g + 8 * (h >> 1), j = j0 + 2 * q + (h & 1);
                if (i >= j) D[i * LDT + j] -= s[h];
            }
        }
        __syncthreads();
    }
    // The 4 diagonal blocks of W, a warp each, a lane per column.
    if (warp < 4) {
        const int p = 32 * warp;
        double w[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) w[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            w[j] *= D[(p + j) * LDT + p + j + 1];
#pragma unroll
            for (int i = 1; i < 32; ++i)
                if (i > j) w[i] -= D[(p + i) * LDT + p + j] * w[j];
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (i >= lane) D[(p + lane) * LDT + p + i + 1] = w[i];
    }
    __syncthreads();
    // Block row I of W left of its diagonal block: W_I = -W_II (L_I W), 32 x 32 I values, as
    // tiles of 16 x 8 (at most 3 per warp).
    for (int I = 1; I < NB / 32; ++I) {
        const int p = 32 * I, tiles = 2 * (p / 8);
        for (int e = warp; e < tiles; e += TH / 32) {
            const int i0 = p + 16 * (e & 1), c0 = 8 * (e >> 1), c = c0 + g;
            double s[4] = {};
            for (int k = c0; k < p; k += 8) {
                const double u[4] = {D[(i0 + g) * LDT + k + q], D[(i0 + g + 8) * LDT + k + q],
                                     D[(i0 + g) * LDT + k + q + 4],
                                     D[(i0 + g + 8) * LDT + k + q + 4]};
                // W[k][c], 0 above its diagonal (where D holds L).
                const double w0 = k + q >= c ? D[c * LDT + k + q + 1] : 0.0;
                const double w1 = k + q + 4 >= c ? D[c * LDT + k + q + 5] : 0.0;
                dmma16(s, u, w0, w1);
            }
#pragma unroll
            for (int h = 0; h < 4; ++h)
                D[(c0 + 2 * q + (h & 1)) * LDT + i0 + g + 8 * (h >> 1) + 1] = s[h];
        }
        __syncthreads();
        double t[3][4] = {};
#pragma unroll
        for (int turn = 0; turn < 3; ++turn) {
            const int e = warp + turn * (TH / 32);
            if (e < tiles) {
                const int i0 = 16 * (e & 1), c = 8 * (e >> 1) + g;
#pragma unroll
                for (int k = 0; k < 32; k += 8) {
                    // W_II[i][k], 0 above its diagonal.
                    double u[4];
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const int i = i0 + g + 8 * (h & 1), kk = k + q + 4 * (h >> 1);
                        u[h] = i >= kk ? -D[(p + kk) * LDT + p + i + 1] : 0.0;
                    }
                    dmma16(t[turn], u, D[c * LDT + p + k + q + 1], D[c * LDT + p + k + q + 5]);
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int turn = 0; turn < 3; ++turn) {
            const int e = warp + turn * (TH / 32);
            if (e < tiles) {
                const int i0 = p + 16 * (e & 1), c0 = 8 * (e >> 1);
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    D[(c0 + 2 * q + (h & 1)) * LDT + i0 + g + 8 * (h >> 1) + 1] = t[turn][h];
            }
        }
        __syncthreads();
    }
    for (int e = tid; e < NB * LDT; e += TH) pair[e] = D[e];
}

// Step 1 of the first diagonal block.
__global__ void __launch_bounds__(TH, 1)
    k_spd_first(int64_t n, int64_t ld, const double* __restrict__ L,
                const double* __restrict__ diag, double* __restrict__ pair,
                unsigned long long* __restrict__ status) {
    extern __shared__ double sm[];
    for (int e = threadIdx.x; e < NB * NB; e += TH) {
        const int i = e % NB, j = e / NB;
        if (i >= j) sm[i * LDT + j] = L[i + (int64_t)j * ld];
    }
    diagonal_block(sm, diag, 0, (int)min((int64_t)NB, n), pair, status);
}

// The products of a panel piece with the diagonal block: the 32 x 16 values (warp w: columns 16w
// to 16w + 15) sum_k X[r][k] M[c][k] over k <= c, M = W (above the diagonal of the pair D) or L
// (on and below it).
template <bool INVERSE>
__device__ __forceinline__ void piece_product(const double* xs, const double* D,
                                              double (&acc)[2][2][4]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int c0 = 16 * warp;
    for (int kk = 0; kk < c0 + 16; kk += 8) {
        double a[2][4], b[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            a[i][0] = xs[(kk + q) * LDP + g + 16 * i];
            a[i][1] = xs[(kk + q) * LDP + g + 16 * i + 8];
            a[i][2] = xs[(kk + q + 4) * LDP + g + 16 * i];
            a[i][3] = xs[(kk + q + 4) * LDP + g + 16 * i + 8];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = kk + q + 4 * h, c = c0 + 8 * j + g;
                b[j][h] = k > c ? 0.0 : INVERSE ? D[k * LDT + c + 1] : D[c * LDT + k];
            }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) dmma16(acc[i][j], a[i], b[j][0], b[j][1]);
    }
}

// Step 2: 32 rows of L below the block (the first blocks) or of V down to the block's own, in
// place: X = A L11^-T as X0 = A W^T and 1 step of refinement, X = X0 + (A - X0 L11^T) W^T, which
// brings the product back to a substitution's accuracy. (Without it the inverse of a 3,000
// unknown cantilever was 20 times further off, 3.7e-10 against 1.8e-11.)
__global__ void __launch_bounds__(TH, 1)
    k_spd_panel(int64_t ld, int64_t b0, double* __restrict__ L, double* __restrict__ V,
                const double* __restrict__ pair) {
    extern __shared__ double sm[];
    double* xs = sm;               // A, then A - X0 L11^T
    double* x0 = sm + NB * LDP;
    double* D = x0 + NB * LDP;
    const int64_t lower = (ld - b0 - NB) / PR, x = blockIdx.x;
    double* X = (x < lower ? L + b0 + NB + x * PR : V + (x - lower) * PR) + b0 * ld;
    for (int e = threadIdx.x; e < NB * LDT / 2; e += TH) copy16(D + 2 * e, pair + 2 * e);
    for (int e = threadIdx.x; e < NB * PR / 2; e += TH) {
        const int r = 2 * (e % (PR / 2)), k = e / (PR / 2);
        copy16(xs + k * LDP + r, X + r + (int64_t)k * ld);
    }
    copy_commit();
    copy_wait<0>();
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // f(row, column, value) for each of the thread's values of the piece.
    auto each = [&](double (&v)[2][2][4], auto f) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    f((lane >> 2) + 16 * i + 8 * (h >> 1),
                      16 * warp + 8 * j + 2 * (lane & 3) + (h & 1), v[i][j][h]);
    };
    double acc[2][2][4] = {}, r1[2][2][4] = {};
    piece_product<true>(xs, D, acc);
    each(acc, [&](int r, int c, double& v) { x0[c * LDP + r] = v; });
    __syncthreads();
    piece_product<false>(x0, D, r1);
    each(r1, [&](int r, int c, double& v) { xs[c * LDP + r] -= v; });
    __syncthreads();
    piece_product<true>(xs, D, acc);
    each(acc, [&](int r, int c, double& v) { X[r + (int64_t)c * ld] = v; });
}

// Tile x of the lower triangle, row by row.
__device__ __forceinline__ void lower_tile(int64_t x, int64_t* bi, int64_t* bj) {
    int64_t i = (int64_t)((sqrt(8.0 * (double)x + 1.0) - 1.0) / 2.0);
    while ((i + 1) * (i + 2) / 2 <= x) ++i;
    while (i * (i + 1) / 2 > x) --i;
    *bi = i;
    *bj = x - i * (i + 1) / 2;
}

// Step 3, and step 1 of the next diagonal block (block 0).
__global__ void __launch_bounds__(TH, 1)
    k_spd_trailing(int64_t n, int64_t ld, int64_t b0, double* __restrict__ L,
                   double* __restrict__ V, const double* __restrict__ diag,
                   double* __restrict__ pair, unsigned long long* __restrict__ status) {
    extern __shared__ double sm[];
    const int64_t t0 = b0 + NB, t = (ld - t0) / NB, nl = t * (t + 1) / 2, x = blockIdx.x;
    const double *A, *B;
    double* C;
    if (x < nl) {
        int64_t bi, bj;
        lower_tile(x, &bi, &bj);
        A = L + t0 + bi * NB + b0 * ld;
        B = L + t0 + bj * NB + b0 * ld;
        C = L + t0 + bi * NB + (t0 + bj * NB) * ld;
    } else {
        const int64_t c = (x - nl) % (b0 / NB + 1), r = (x - nl) / (b0 / NB + 1);
        A = V + c * NB + b0 * ld;
        B = L + t0 + r * NB + b0 * ld;
        C = V + c * NB + (t0 + r * NB) * ld;
    }
    // The 128 products are summed from 0 and then taken off the tile: 1 rounding at the size of
    // the tile's values per step. (Started from the tile, 128 roundings: the inverse of the 3,000
    // unknown cantilever 3.7e-10 off in place of 1.8e-11.)
    double acc[4][4][4] = {};
    tile_product(A, B, ld, NB, sm, acc);
    if (x > 0) {
        take_off(acc, C, ld);
        return;
    }
    each_value(acc, [&](int r, int c, double& v) {
        if (r >= c) sm[r * LDT + c] = C[r + (int64_t)c * ld] - v;
    });
    diagonal_block(sm, diag, t0, (int)max((int64_t)0, min((int64_t)NB, n - t0)), pair, status);
}

// A^-1 = V V^T: V[i][k] = 0 for k < i, so the sum of a tile starts at its rows. The long sums
// come first.
__global__ void __launch_bounds__(TH, 1)
    k_spd_gram(int64_t n, int64_t ld, const double* __restrict__ V, double* __restrict__ X) {
    extern __shared__ double sm[];
    int64_t bi, bj;
    lower_tile(blockIdx.x, &bi, &bj);
    const int64_t i0 = bi * NB, j0 = bj * NB;
    double acc[4][4][4] = {};
    tile_product(V + i0 + i0 * ld, V + j0 + i0 * ld, ld, (int)(ld - i0), sm, acc);
    each_value(acc, [&](int r, int c, double& v) {
        const int64_t i = i0 + r, j = j0 + c;
        if (i < n && j <= i) {
            X[i + j * n] = v;
            X[j + i * n] = v;
        }
    });
}

// The identity on the padding's diagonal of L, and on V's.
__global__ void k_spd_identity(int64_t n, int64_t ld, double* __restrict__ L,
                               double* __restrict__ V) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= ld) return;
    if (i >= n) L[i + i * ld] = 1.0;
    V[i + i * ld] = 1.0;
}

}  // namespace

void spd_factor(int64_t n, double* L, double* V, const double* diag, double* pair,
                unsigned long long* status, cudaStream_t s) {
    const int64_t ld = spd_padded(n);
    FG_CUDA(cudaFuncSetAttribute(k_spd_first, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)DIAG_SMEM));
    FG_CUDA(cudaFuncSetAttribute(k_spd_panel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)PANEL_SMEM));
    FG_CUDA(cudaFuncSetAttribute(k_spd_trailing, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)STEP_SMEM));
    FG_CUDA(cudaMemsetAsync(V, 0, (size_t)(ld * ld) * sizeof(double), s));
    k_spd_identity<<<(unsigned)(ld / NB), NB, 0, s>>>(n, ld, L, V);
    k_spd_first<<<1, TH, DIAG_SMEM, s>>>(n, ld, L, diag, pair, status);
    for (int64_t b0 = 0; b0 < ld; b0 += NB) {
        k_spd_panel<<<(unsigned)(ld / PR), TH, PANEL_SMEM, s>>>(ld, b0, L, V, pair);
        const int64_t t = (ld - b0) / NB - 1;
        if (t > 0)
            k_spd_trailing<<<(unsigned)(t * (t + 1) / 2 + (b0 / NB + 1) * t), TH, STEP_SMEM, s>>>(
                n, ld, b0, L, V, diag, pair, status);
    }
    FG_CHECK_LAUNCH();
}

void spd_gram(int64_t n, const double* V, double* inv, cudaStream_t s) {
    const int64_t ld = spd_padded(n), t = ld / NB;
    FG_CUDA(cudaFuncSetAttribute(k_spd_gram, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TILE_SMEM));
    k_spd_gram<<<(unsigned)(t * (t + 1) / 2), TH, TILE_SMEM, s>>>(n, ld, V, inv);
    FG_CHECK_LAUNCH();
}

}  // namespace femgpu
