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
    const float *q, *dinv;
    const double* b64;    // right-hand side (init) or FP64 residual (restart), by equation
    const int* aeq;       // padded node blocks: equation of every component, else null
    CGScal* S;
    double* part;
    double tol, drop;     // init
    int max_iter;
};

// the FP32 matrix: sliced-ELL 3x3 blocks, or scalar CSR
struct CzMat {
    const int *soff, *swid, *rowptr, *col;
    const float* val;
};

// support points, boxes and row lists for the current pattern; c->cz.ok says
// whether the two-level solve is available
int coarse_plan(isl_ctx* c, int nc, int64_t nrow);
// Galerkin blocks and the dense inverse for the current assembly
int coarse_numeric(isl_ctx* c, const CzMat& A);
void coarse_args(const isl_ctx* c, CzIter& a);
// update (or start, or restart) and coarse correction: two launches
void launch_coarse(const isl_ctx* c, cudaStream_t st, const CzIter& a, int mode);
void launch_coarse_dir(const isl_ctx* c, cudaStream_t st, int n, const float* z, float* p, const CGScal* S);

}  // namespace isl
