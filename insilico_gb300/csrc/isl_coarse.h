// Two-level preconditioner of the mixed CG: interface between isl_coarse.cu
// (plan, numeric setup, kernels) and the solve in isl_solver.cu.
#pragma once

#include "isl_internal.h"

namespace isl {

enum { CZ_UPDATE = 0, CZ_INIT = 1, CZ_RESTART = 2 };

// arguments of the iteration kernels
struct CzIter {
    const float4* lnode;  // rows listed by sub-aggregate: scaled position, row (and mask)
    const int* sofs;      // first list entry of every sub-aggregate
    const float* dsub;    // inverse blocks of the sub-aggregates
    const float* ainv;    // dense inverse [ndp][ndp]
    float* rc;            // P^T r [ndp]
    int ndp;
    float *x, *r, *z;
    const float *p1, *p2; // direction (p2: the buffer of even iteration counts, null when there is one)
    float* pz;            // direction buffer zeroed at the start
    const float *q;
    const float* dinv;    // inverse diagonal (blocks) in list order, [1 or 9][nrow]
    int nrow;
    const double* b64;    // right-hand side (init) or FP64 residual (restart), by equation
    const int* aeq;       // padded node blocks: equation of every component, else null
    CGScal* S;
    double* part;
    double tol, drop;     // init
    int max_iter, max_gap;
};

// the FP32 matrix: sliced-ELL 3x3 blocks, scalar sliced ELL, or scalar CSR
struct CzMat {
    const int *soff, *swid, *rowptr, *col;
    const float* val;
};

// arguments of the scalar product q = A p
struct CzSpmv {
    const int *bnd, *soff;  // first slice of every CTA; first entry of every slice
    const float *val, *p;
    float* q;
    CGScal* S;
    double* part;
    int nrow;
};

// support points, boxes and row lists for the current pattern; c->cz.ok says
// whether the two-level solve is available.  Scalar systems get their
// aggregate-ordered sliced-ELL copy, or, with ncta > 0, the (block) CSR copy
// of the one-cluster solve and its distribution over ncta CTAs.
int coarse_plan(isl_ctx* c, int nc, int64_t nrow, int ncta);
// for the current assembly: values of the aggregate-ordered copy, inverse
// diagonal of scalar rows (in that order), Galerkin blocks, dense inverse
int coarse_numeric(isl_ctx* c, bool csr, float* dinv);
// gives the plan's memory back and leaves this pattern to the one-level solve:
// after one of the calls here returned ISL_ERR_NOMEM
void coarse_drop(isl_ctx* c);
// a batch's result records, cleared
int coarse_results(isl_ctx* c);
void coarse_args(const isl_ctx* c, CzIter& a);
// update (or start, or restart) and coarse correction: two launches
void launch_coarse(const isl_ctx* c, cudaStream_t st, const CzIter& a, int mode);
// Iterations without a reliable update (a residual ten times smaller) after which
// a solve of at most max_iter of them is given up: a healthy one takes some
// hundred, and what FP32 directions cannot bring further ends as the one-level
// solve does.  30^3 cells, 20 times thinner than wide, which neither solves to
// 1e-10: 5.0 s with the limit of neq / 4 iterations alone, 4.6 s so, 4.5 s one-level.
inline int coarse_gap(int max_iter) { return max_iter / 8 > 1000 ? max_iter / 8 : 1000; }
// the whole solve in one launch, a thread-block cluster or a cooperative grid
// of z.ncta CTAs (after coarse_plan with ncta > 0 and coarse_numeric): work
// holds 3 vectors, the FP64 iterate goes to x64 and the record's fin, iters
// and residuals to c->dscal; on a batch, every instance of the class z.cls[cls] in
// a cluster of its own, or the instance z.big[big] in a grid, results in z.res
int coarse_cluster_fits(const isl_ctx* c, bool grid);
cudaError_t launch_coarse_cluster(isl_ctx* c, bool grid, cudaStream_t st, float* work, const float* dinv, double* x64, double tol, double drop,
                                  int max_iter, int big = -1, int cls = 0);
// scalar product (kind 102, 104, 108: 4, 8 or 12 slots in flight), and its CTAs' runs of slices (once per pattern)
int coarse_spmv_plan(isl_ctx* c);
void launch_coarse_spmv(const isl_ctx* c, int kind, cudaStream_t st, const CzSpmv& m);
void launch_coarse_dir(const isl_ctx* c, cudaStream_t st, int n, const float* z, float* p, const CGScal* S);

}  // namespace isl
