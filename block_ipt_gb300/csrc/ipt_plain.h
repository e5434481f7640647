// ipt_plain.h - FP64 plain-IPT drivers behind the reference ABI (internal).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "kernels.cuh"
#include "oz_product.h"

namespace iptgb {

// One application of the IPT map X' = F(X) in FP64, plus (H X)_jj.
struct Fp64Operator {
    virtual ~Fp64Operator() = default;
    // Before the first step from an n x k block X with diagonal d.
    virtual int start(const double *X, int k, const double *d) = 0;
    // Xn = F(X); with want_norms the step leaves ||Xn - X||_F, ||X||_F in ns->norms.
    virtual int step(const double *X, double *Xn, const double *d, int want_norms,
                     NormScratch *ns) = 0;
    // The same, where the norms may reach ns->norms only with the next step or
    // with flush_norms().
    virtual int step_ahead(const double *X, double *Xn, const double *d, NormScratch *ns)
    {
        return step(X, Xn, d, 1, ns);
    }
    virtual int flush_norms() { return IPT_CUDA_SUCCESS; }
    // waits for the steps and reports one that failed (its block is NaN)
    virtual int check() { return IPT_CUDA_SUCCESS; }
    // values[j] = (H X)_jj.
    virtual int diag_values(const double *X, double *values) = 0;
};

// Dense H: Delta X by the 56-bit digit-slice product on the tensor cores
// (k_oz.cu), whose consumer applies the map.  It replaces a split-K FP64 SIMT
// product (GB300 runs FP64 FMAs at 1/64 of the FP32 rate; on a matrix of few
// row blocks most SMs stood idle as well): a step takes 165 us instead of 3.7
// ms at n = 8192, k = 32, 27 us instead of 105 us at n = 1024, k = 8, so no
// size keeps the old one for its time; 0.33 instead of 6.1 ms with all n = 1501
// columns.
//
// Its error: in the 2-norm it is the smaller one (after 12 steps at n = k =
// 1501 8e-16 against 7e-14: the diagonal, which the FP64 product carried
// through y and the map took off again, is left out).  Entry by entry, a block
// of 128 columns adds up to 128 2^-54 max_l |Delta_il| max_l |X_lc| (l in the
// block) to an entry of Delta X, where FP64 FMAs stay relative to the terms
// themselves.  So a matrix with rows whose entries span many binades within a
// block (graded ones, sparse or banded ones stored as dense, couplings that
// decay within tens of rows) keeps the FP64 FMAs, found out when the digits are
// laid out (OzMatrix::wide): every entry of the vectors is then as accurate as
// theirs.
struct DenseFp64Operator final : Fp64Operator {
    OzMatrix own;
    const OzMatrix *matrix = &own;
    OzProduct product;
    DeviceBuffer<double> g;  // n x k gap reciprocals
    const double *H = nullptr;
    int n = 0, k = 0;
    int slices = 7;  // 0: FP64 FMAs, where the environment asks for them
    cudaStream_t stream = nullptr;
    // scans H (column-major n x n); d (optional) receives its diagonal
    int bind(const double *H, int n, double *d, cudaStream_t s);
    // the same on a matrix the caller has scanned and laid out (and keeps)
    void share(const OzMatrix *scanned, cudaStream_t s);
    int start(const double *X, int k, const double *d) override;
    int step(const double *X, double *Xn, const double *d, int want_norms,
             NormScratch *ns) override;
    int step_ahead(const double *X, double *Xn, const double *d, NormScratch *ns) override;
    int flush_norms() override { return product.flush_norms(); }
    int check() override { return product.check(); }
    int diag_values(const double *X, double *values) override;
};

struct CsrFp64Operator final : Fp64Operator {
    const int *row_ptr = nullptr;
    const int *col_ind = nullptr;
    const double *vals = nullptr;
    int n = 0, k = 0;
    double *Y = nullptr;  // n * k
    cudaStream_t stream = nullptr;
    int start(const double *, int, const double *) override { return IPT_CUDA_SUCCESS; }
    int step(const double *X, double *Xn, const double *d, int want_norms,
             NormScratch *ns) override;
    int diag_values(const double *X, double *values) override;
};

// Scratch owned by a solve: norm reduction slots + readback.
struct SolveScratch {
    NormScratch ns;
    // the read-backs land in pageable memory: each is followed by a stream
    // synchronisation anyway, and a pinned allocation (with the device-wide
    // synchronisation of its release) per solve cost more than it saved
    double host_norms[2] = {0.0, 0.0};
    std::vector<double> host_hist;
    int init(size_t max_elems, cudaStream_t stream);
    // for an n x k block, whose reductions may take whole blocks per column
    int init(int n, int k, cudaStream_t stream);
    void release(cudaStream_t stream);
    // zeroed history for up to `steps` steps with the device-side stop at tol
    int arm_history(int steps, double tol, cudaStream_t stream);
    // the first `count` history entries: *stopped_at = first step that met
    // the tolerance (-1: none), *rel = its ||delta||/||X|| (else the last
    // entry's); synchronises the stream
    int read_history(int count, int *stopped_at, double *rel, cudaStream_t stream);
};

// The reference's plain IPT loop (IPT_C_GPU/src/ipt_cuda.cu:1644-1703):
// X_a holds the start block on entry; on success *X_final points at the
// buffer (X_a or X_b) holding the returned block.  In tolerance mode the loop
// stops once ||F(X)-X||_F / ||X||_F <= tol and returns F(X).
int run_plain_ipt(Fp64Operator &op, int n, int k, const double *d, int maxiter, double tol,
                  int use_tol, double *X_a, double *X_b, double **X_final,
                  int *iterations_done, double *fixed_point_residual, SolveScratch *scratch,
                  cudaStream_t stream);

int device_sm_count();

}  // namespace iptgb
