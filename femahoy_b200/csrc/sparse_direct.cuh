// The sparse direct solver on the device: a multifrontal Cholesky factor P A P^T = L L^T over
// the supernodes of the host analysis (symbolic.hpp), as the reference factors its "direct"
// systems (cholesky.rs:44-167; the order of order.rs, the supernodes of symbolic.rs), and the
// two triangular solves.
//
// Layout. Each supernode s owns a dense frontal matrix F_s of m_s x m_s doubles (column-major,
// its rows R_s) while it is factored: its first k_s columns become the columns of L, and its
// trailing block is the update matrix (Schur complement) that its parent takes. The entries of A
// are scattered into all fronts at once; then the fronts are done level by level in the
// supernode tree (height 0 = leaves), so every child is factored before its parent:
//   1. extend-add: each child's update matrix is added into its parent's front at the parent's
//      rows (relative indices found on the host), 1 launch per child rank, so the sums into a
//      parent are made in a fixed order (no atomics; the factor is reproducible bit for bit);
//   2. partial Cholesky of the k_s pivot columns: fronts of at most 128 rows in shared memory, 1
//      block each (all the level's small fronts in 1 launch); a larger front by panels of 32
//      columns (the diagonal block and the panel's rows in 1 kernel, then the trailing update
//      F22 -= L21 L21^T on the FP64 tensor cores, mma.sync m8n8k4 f64, in 64 x 64 tiles).
// A pivot at or below PIVOT = 1e-10 of the column's diagonal of A (cholesky.rs:22, 176-181) is
// recorded (the smallest column; every front with no failed descendant is still checked, so
// this is the reference's first failing column) and the factor fails with the reference's text.
// Then the fronts give way to the form of the solves: each supernode's G = [W; -L21 W] with
// W = L11^-1 (m_s x k_s), so that a supernode's step is 1 product in either direction and splits
// over as many blocks as it has rows (forward) or columns (backward). The solves run level by
// level: forward up the tree, backward from the root down. The products round as W does, not as
// a substitution: on the direct solves of the test systems the true residuals stay those of the
// substitution (4.1e-11 against 4.3e-11 on a 36,300-unknown P2 beam, 1.4e-15 on a 32^3 heat
// cube).
#pragma once
#include <string>
#include <vector>

#include "common.cuh"
#include "hierarchy.hpp"
#include "symbolic.hpp"

namespace femgpu {

// A part of a supernode's step in the solves: its panel G (offset g, m rows, k columns, leading
// dimension ld), where its rows (z) and columns (j0) start, and the part: 32 rows from `at`
// (forward), or `cols` columns from `at` (backward).
struct SolveTask {
    int64_t g, z, j0;
    int ld, m, k, at, cols, pad;
};
// A block's tasks: `count` from `task`, each with `warps` of the block's 16 warps.
struct SolveBlock {
    int task, count, warps;
};

class SparseFactor {
   public:
    // Analyses and factors `a` (host CSR, both triangles) in the nested dissection order of the
    // unknowns' coordinates `xyz` (3 per unknown).
    void factor(const HostCsr& a, const double* xyz, cudaStream_t s);
    // x = A^-1 b in FP64, device arrays of n values (x may not alias b; both double, or both float
    // and converted on the way). `pdl`: programmatic dependent launches.
    template <class TB, class TX>
    void solve(const TB* b, TX* x, bool pdl, cudaStream_t s);
    int64_t n() const { return n_; }
    // The kernels that 1 solve launches.
    size_t solve_launches() const;
    size_t bytes() const;
    std::string describe() const;
    uint64_t entries() const { return entries_; }

   private:
    void pack(cudaStream_t s);

    int64_t n_ = 0, ns_ = 0, height_ = 0, large_fronts_ = 0;
    uint64_t entries_ = 0;
    double flops_ = 0.0;
    size_t front_values_ = 0;
    // Per supernode (device): first column, row list, front offset.
    DevBuf<int64_t> perm_, first_, rows_ptr_, foff_;
    DevBuf<uint32_t> rows_;
    DevBuf<double> fronts_;  // until the factor is packed
    // The G panels end to end; the forward solution and the backward one (both in the
    // elimination order); the children's updates (slots) with each row's first slot and the
    // slot that each update row writes in its parent.
    DevBuf<double> g_, y_, xs_, slot_;
    DevBuf<uint32_t> slot_ptr_, dst_;
    DevBuf<SolveBlock> forward_blocks_, backward_blocks_;
    DevBuf<SolveTask> forward_tasks_, backward_tasks_;
    std::vector<int64_t> forward_at_, backward_at_;  // per height: offsets into the blocks
    // Host: the supernodes of each height, their rows and columns, and where their rows, columns
    // and fronts start.
    std::vector<std::vector<int64_t>> levels_;
    std::vector<int64_t> m_, k_, host_zoff_, host_first_, host_foff_;
};

}  // namespace femgpu
