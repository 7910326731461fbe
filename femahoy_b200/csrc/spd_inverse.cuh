// The inverse of a dense SPD matrix on the device, in FP64 on the tensor cores.
//
// A = L L^T and W = L^-1 are formed together, 128 columns at a time, then A^-1 = W^T W. Step b:
//   1. the 128 x 128 diagonal block is factored and inverted in shared memory by 1 block;
//   2. the panels: the rows of L below it and the rows of V = W^T so far, each 32 x 128 piece
//      times the inverse of the diagonal block's factor, with 1 step of refinement;
//   3. the trailing update, 128 x 128 tiles with 128 inner terms: the lower tiles of A's trailing
//      block by L L^T and the tiles of V right of the panel by V L^T, in 1 launch. Its first
//      block updates the next diagonal block and goes on to step 1 of b + 1 there, so that the
//      serial factor of a diagonal block runs beside the other tiles' products.
// V is kept in place of W because every product is then C -= A B^T over operands whose rows are
// contiguous. The matrices are padded to a multiple of 128 with the identity, so that no tile
// has an edge.
//
// What bounds it: n^3 operations (118 Gflop at n = 4,913) at the FP64 rate, and the serial factor
// of each diagonal block. On B200 at n = 4,000: trailing updates 3.1 ms (100 us each: 3 waves of
// tiles, 20-25 us per tile, the diagonal block's factor 64 us beside them), panels 0.5 ms, V V^T
// 0.85 ms (25 Tflop/s): 4.5 ms. By panels of 32 columns with W formed afterwards the inverse of
// the 128^3 heat cube's 4,913 unknowns took 23 ms, of which 0.8 us per column went to the panels'
// diagonal blocks alone, and every rank-32 update read and wrote the whole trailing matrix. The
// products sum 128 terms before they meet the matrix, so it rounds no more often than before. 1
// product with the inverse of 18 P1 cantilevers of 1,380 to 2,700 unknowns (3 right sides each, off
// an extended precision solution, geometric means; before in brackets): Poisson ratios of 0.25 to
// 0.35 1.9e-12 (2.9e-12), stiffness jumps of 1e6 7.9e-12 (8.5e-12), a ratio of 0.4999 1.4e-10
// (0.8e-10; a Cholesky factor with substitutions on the host 4.1e-10).
#pragma once
#include <cstdint>

#include "common.cuh"

namespace femgpu {

constexpr int SPD_BLOCK = 128;
constexpr int SPD_PAIR = SPD_BLOCK * (SPD_BLOCK + 4);

inline int64_t spd_padded(int64_t n) { return (n + SPD_BLOCK - 1) / SPD_BLOCK * SPD_BLOCK; }

// L: the lower triangle of A in the first n rows and columns of a column-major array of leading
// dimension spd_padded(n), zero elsewhere (overwritten); V: an array of the same size; diag: the
// n diagonal entries of A; pair: SPD_PAIR values. A pivot at or below 1e-10 of its column's
// diagonal records the column in *status (an atomic minimum; the caller sets it to ~0 first).
// spd_factor queues steps 1-3, spd_gram the product V V^T into inv (n x n, both halves, exactly
// symmetric).
void spd_factor(int64_t n, double* L, double* V, const double* diag, double* pair,
                unsigned long long* status, cudaStream_t s);
void spd_gram(int64_t n, const double* V, double* inv, cudaStream_t s);

}  // namespace femgpu
