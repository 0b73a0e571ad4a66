// Row-major multivector products with fused epilogues (spmm_tc.cu), used by
// the multi-right-hand-side cycle (multirhs.cu).
#pragma once

#include "amgt_internal.cuh"

namespace amgt {

// X: the multiplied vectors, Y: the result, both rows x nvec; w = alpha.
enum {
    MV_SPMM = 0,     // Y = alpha A X + beta Y
    MV_RESID = 1,    // Y = F - A X
    MV_RESID0 = 2,   // Y = F - A u, u = w X ./ l1 (X = F: the residual after a sweep from zero)
    MV_CORRECT = 3,  // Y = A X + w F ./ l1 (the prolonged correction on that sweep's result)
    MV_JACOBI = 4,   // Y = X + w (F - A X) ./ l1; with part, partials of F . Y
    MV_DOT = 5       // Y = A X; partials of X . Y
};
struct MvArgs {
    int m, n, brow, nvec;
    int split;  // parts of a block row
    const int *ptr, *idx;
    const uint16_t *map;
    const void *val;
    double alpha, beta;
    const double *X, *F, *inv_l1;
    double *Y;
    double *part;  // mv_apply_grid x 32: partials per CTA and column
};
int mv_apply_grid(const amgt_bsr *A, int nvec, int sm_count);
int mv_apply(int prec, int epi, const amgt_bsr *A, int nvec, const MvArgs &a, cudaStream_t s, int sm_count);

}  // namespace amgt
