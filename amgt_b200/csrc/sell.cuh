// Sliced copies of the cycle's operators (internal; sell.cu).
#pragma once

#include <vector>

#include "amgt_internal.cuh"

namespace amgt {

// An operator of the AMG cycle in slices: a warp's worth of rows (32 >> log_t
// of them, 1 << log_t lanes each) with only the stored entries, padded to the
// slice's longest row with zeros at the row's own last column.  Step k of slice
// s holds entry (k << log_t) + t of row i at 32 (hdr[s].x + k) + (i << log_t) +
// t: the column minus hdr[s].z (16 bits) or the column (idx32) and the value,
// in the storage types that the cycle's precisions read.
struct SellMat {
    int m = 0, n = 0, nslices = 0, log_t = 0;
    bool idx32 = false, holes = false;  // holes: some row has no entry
    int4 *hdr = nullptr;  // device [nslices]: first step, steps, column base, mask of non-empty rows
    void *idx = nullptr;
    void *val[4] = {nullptr, nullptr, nullptr, nullptr};  // fp64, fp32, fp16, bf16
};

// Storage type (index into SellMat::val) of a value mode (spmv_common.cuh).
int sell_storage(int mode);
// True when S holds the values that products at `mode` read.
bool sell_has(const SellMat &S, int mode);

// One operator to copy: storages: bit k set for val[k].
struct SellJob {
    const amgt_bsr *A;
    unsigned storages;
    SellMat *out;
};
// True when a sliced copy of A pays: see sell.cu.
bool sell_wanted(const amgt_bsr *A);
// Two steps, so that one host read-back (the caller's) sizes every copy:
// measure launches the pass that sizes the slices, writing per job the
// total steps, the widest column span above 65,535, the longest slice above 64
// steps and whether a row is empty to meas[kSellMeas j ...] (device, zeroed by
// the caller); fill allocates and fills the copies with
// those numbers on the host.  A copy that would not pay (see there), or for
// which the allocator has no memory, is left out (out->hdr is null).
constexpr int kSellMeas = 4;
int sell_measure(const std::vector<SellJob> &jobs, int64_t *meas, cudaStream_t s, int sm_count);
int sell_fill(const std::vector<SellJob> &jobs, const int64_t *meas_host, cudaStream_t s, int sm_count);
void sell_free(SellMat &S, cudaStream_t s);

// Products at a value mode; the contracts of spmv.cu's fused forms.
int sell_spmv(const SellMat &S, int mode, double alpha, const double *x, double beta, double *y, cudaStream_t s,
              int sm_count);
int sell_residual(const SellMat &S, int mode, const double *f, const double *u, double *r, cudaStream_t s,
                  int sm_count);
int sell_jacobi(const SellMat &S, int mode, const double *inv_l1, double w, const double *f, const double *u,
                double *u_out, cudaStream_t s, int sm_count);
int sell_restrict_jacobi0(const SellMat &S, int mode, const double *t, double *f, const double *inv_l1, double w,
                          double *u, cudaStream_t s, int sm_count);
// partial: sell_dot_grid entries (the grid does not depend on the mode)
int sell_dot_grid(const SellMat &S, int sm_count);
int sell_dot(const SellMat &S, int mode, const double *u, double *out, double *partial, cudaStream_t s, int sm_count);

}  // namespace amgt
