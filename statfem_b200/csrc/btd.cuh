// Direct solve of symmetric positive definite block-tridiagonal systems: the
// plan and launch interface of btd.cu.
#pragma once

#include "common.cuh"

namespace sfc {

// entries of a row that couple it to the line before and after it, and to its own line
constexpr int kBtdSide = 4, kBtdMid = 8;
constexpr int kBtdCols = 32;  // right-hand sides of a column tile

struct BtdArgs {
    // operator (CSR, FP64); instance i owns dofs [row0[i], row0[i + 1]) cut
    // into lines of line[i] dofs, coupled to the neighbouring lines only
    const int32_t *rp, *col;
    const double *a;
    int n_inst;
    const int64_t *row0;
    const int32_t *line, *order;
    int64_t N;
    // per dof: padded entries towards the previous line, the next line and its own line
    int16_t *lc, *uc, *mc;
    double *lv, *uv, *mv;
    // inverse blocks and coupling scratch of a cluster (slot)
    double *X, *Y;
    int64_t xstride, ystride;
    // right-hand sides and solutions, interleaved [dof][ld]
    const double *B;
    double *U;
    int ld, ncols;
    int *queue;
    int *bad;    // per instance: 1 where a pivot was not a positive number the reciprocal takes
    int chain;   // CTAs per elimination chain; a cluster has two chains
    int lmax;    // longest line
};

// Looks whether the system's pattern has the form above and sizes the
// workspace; false when the direct solve does not apply.
bool btd_plan(sfc_ctx *ctx, BtdPlan &p, const int32_t *rp, const int32_t *col, int64_t N, int n_inst,
              const int64_t *row0, const int32_t *line, const int32_t *order, bool keep_blocks);
BtdArgs btd_args(BtdPlan &p, const int32_t *rp, const int32_t *col, const double *a);
// factor and solve every instance (32 columns each), one cluster per instance
void btd_launch_batch(sfc_ctx *ctx, const BtdPlan &p, const BtdArgs &a, cudaStream_t st);
// one system: the inverse blocks, then any number of columns
void btd_launch_factor(sfc_ctx *ctx, const BtdPlan &p, const BtdArgs &a);
void btd_launch_solve(sfc_ctx *ctx, const BtdPlan &p, const BtdArgs &a);
// Whether the system's pattern has the form (planned on the first call), and an
// estimate of a solve for nrhs columns in us (with the factor, unless it is there)
bool btd_applies(sfc_system *s);
double btd_estimate(const sfc_system *s, int nrhs);
// S X = B of a system whose operator is built, refined with FP64 residuals
// where the first solution misses tol; false (X undefined) where the
// elimination does not apply, the operator is not positive definite or a
// column's true residual still misses tol.  `recurrence`: in place of a solver
// that stops by its recurrence residual, which does not see the rounding of
// the true one; a residual at that rounding is then accepted too.
bool btd_solve_system(sfc_system *s, const double *B, double *X, int nrhs, int ld, double tol, bool recurrence,
                      double *max_rel);

}  // namespace sfc
