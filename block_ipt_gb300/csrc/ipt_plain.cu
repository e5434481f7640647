// ipt_plain.cu - FP64 plain-IPT driver loop.
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "ipt_plain.h"
#include "thread_slots.h"

namespace iptgb {

int device_sm_count()
{
    int dev = 0;
    int sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        sms <= 0) {
        return 148;
    }
    return sms;
}

int DenseFp64Operator::bind(const double *H_, int n_, double *d, cudaStream_t s)
{
    H = H_;
    n = n_;
    stream = s;
    slices = fp64_fma_wanted() ? 0 : 7;
    if (slices == 0) {
        own.reference(H, n);
        return d != nullptr ? launch_extract_diagonal(H, n, n, d, s) : IPT_CUDA_SUCCESS;
    }
    IPTGB_CHECK(own.scan_rows(H, n, d, s));
    return own.build_words(7, s);
}

void DenseFp64Operator::share(const OzMatrix *scanned, cudaStream_t s)
{
    matrix = scanned;
    H = scanned->H;
    n = scanned->n;
    stream = s;
    slices = scanned->wide ? 0 : 7;
}

int DenseFp64Operator::start(const double *X, int k_, const double *d)
{
    k = k_;
    IPTGB_CHECK(product.bind(matrix, d, slices, stream));
    if (g.count < (size_t)n * k) IPTGB_CHECK(g.alloc((size_t)n * k, stream));
    IPTGB_CHECK(launch_gap_reciprocals(d, n, k, g.ptr, stream));
    IPTGB_CHECK(product.begin(X, k));
    IPTGB_CHECK(own.settle(stream));
    if (slices == 0 || !matrix->wide) return IPT_CUDA_SUCCESS;
    slices = 0;
    IPTGB_CHECK(product.bind(matrix, d, slices, stream));
    return product.begin(X, k);
}

int DenseFp64Operator::step(const double *X, double *Xn, const double *d, int want_norms,
                            NormScratch *ns)
{
    (void)d;
    return product.step(X, g.ptr, Xn, want_norms, ns);
}

int DenseFp64Operator::step_ahead(const double *X, double *Xn, const double *d, NormScratch *ns)
{
    (void)d;
    return product.step(X, g.ptr, Xn, 1, ns, nullptr, true);
}

int DenseFp64Operator::diag_values(const double *X, double *values)
{
    return launch_dense64_diag_values(H, n, n, X, k, values, stream);
}

int CsrFp64Operator::step(const double *X, double *Xn, const double *d, int want_norms,
                          NormScratch *ns)
{
    {
        KernelTimerScope timer(kProfCsrProduct, stream);
        IPTGB_CHECK(launch_csr64_spmm(row_ptr, col_ind, vals, n, X, k, Y, stream));
    }
    KernelTimerScope timer(kProfFp64Update, stream);
    return launch_ipt_update_from_y(Y, n, k, X, d, Xn, want_norms, ns, stream);
}

int CsrFp64Operator::diag_values(const double *X, double *values)
{
    return launch_csr64_diag_values(row_ptr, col_ind, vals, n, X, k, values, stream);
}

int SolveScratch::init(size_t max_elems, cudaStream_t stream)
{
    const int slots = blocks_for(max_elems);
    IPTGB_CUDA(device_malloc((void **)&ns.partials, (size_t)slots * sizeof(double2), stream));
    // [counter u32 | pad][norms double x2]
    IPTGB_CUDA(device_malloc((void **)&ns.counter, 32, stream));
    ns.norms = (double *)((char *)ns.counter + 16);
    ns.capacity = slots;
    IPTGB_CUDA(cudaMemsetAsync(ns.counter, 0, 16, stream));
    return IPT_CUDA_SUCCESS;
}

int SolveScratch::init(int n, int k, cudaStream_t stream)
{
    return init((size_t)blocks_for((size_t)n) * kThreads * (size_t)k, stream);
}

int SolveScratch::arm_history(int steps, double tol, cudaStream_t stream)
{
    if (steps > ns.hist_cap) {
        if (ns.hist != nullptr) cudaFreeAsync(ns.hist, stream);
        ns.hist = nullptr;
        ns.hist_cap = 0;
        IPTGB_CUDA(device_malloc((void **)&ns.hist, 2 * (size_t)steps * sizeof(double), stream));
        ns.hist_cap = steps;
    }
    IPTGB_CUDA(cudaMemsetAsync(ns.hist, 0, 2 * (size_t)steps * sizeof(double), stream));
    ns.step = 0;
    ns.stop_tol = tol;
    return IPT_CUDA_SUCCESS;
}

int SolveScratch::read_history(int count, int *stopped_at, double *rel, cudaStream_t stream)
{
    host_hist.resize(2 * (size_t)count);
    if (count > 0) {
        IPTGB_CUDA(cudaMemcpyAsync(host_hist.data(), ns.hist, 2 * (size_t)count * sizeof(double),
                                   cudaMemcpyDeviceToHost, stream));
    }
    IPTGB_CUDA(cudaStreamSynchronize(stream));
    *stopped_at = -1;
    *rel = NAN;
    const double t2 = ns.stop_tol * ns.stop_tol;
    for (int i = 0; i < count; ++i) {
        const double d2 = host_hist[2 * (size_t)i], x2 = host_hist[2 * (size_t)i + 1];
        *rel = sqrt(d2) / sqrt(x2);
        if (x2 > 0.0 && d2 <= t2 * x2) {
            *stopped_at = i;
            break;
        }
    }
    return IPT_CUDA_SUCCESS;
}

void SolveScratch::release(cudaStream_t stream)
{
    if (ns.partials != nullptr) {
        cudaFreeAsync(ns.partials, stream);
    }
    if (ns.counter != nullptr) {
        cudaFreeAsync(ns.counter, stream);
    }
    if (ns.hist != nullptr) {
        cudaFreeAsync(ns.hist, stream);
    }
    ns = NormScratch();
}

namespace {

// Per host thread: two page-locked slots of two norms each that the update
// kernels of alternate steps write directly (taken on the thread's first
// tolerance-stopped solve and handed on to another thread when it ends).
constexpr int kNormSlots = 2;

double *make_norm_slots()
{
    void *p = nullptr;
    if (cudaHostAlloc(&p, 2 * kNormSlots * sizeof(double), cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return static_cast<double *>(p);
}

double *pinned_norm_slots() { return ThreadSlots<double>::mine(make_norm_slots); }

// A NaN no kernel produces marks a slot as not yet written.
constexpr uint64_t kNormPending = 0x7FF45EED00000001ULL;

void arm_slot(volatile uint64_t *slot)
{
    slot[0] = kNormPending;
    slot[1] = kNormPending;
}

bool slot_written(const volatile uint64_t *slot)
{
    return slot[0] != kNormPending && slot[1] != kNormPending;
}

// Waits for a slot without a call into the driver per step; the stream is
// queried now and then so that a failed launch ends the wait.
int wait_slot(const volatile uint64_t *slot, cudaStream_t stream)
{
    for (unsigned int polls = 1; !slot_written(slot); ++polls) {
        if ((polls & 0x3FFFu) != 0) continue;
        const cudaError_t e = cudaStreamQuery(stream);
        if (e == cudaErrorNotReady) continue;
        if (e == cudaSuccess && slot_written(slot)) break;
        fprintf(stderr, "ipt_gb300: IPT step did not finish: %s\n", cudaGetErrorString(e));
        return IPT_CUDA_CUDA_ERROR;
    }
    return IPT_CUDA_SUCCESS;
}

}  // namespace

int run_plain_ipt(Fp64Operator &op, int n, int k, const double *d, int maxiter, double tol,
                  int use_tol, double *X_a, double *X_b, double **X_final,
                  int *iterations_done, double *fixed_point_residual, SolveScratch *scratch,
                  cudaStream_t stream)
{
    (void)n;
    double *X[2] = {X_a, X_b};  // step i reads X[i % 2] and writes the other
    IPTGB_CHECK(op.start(X_a, k, d));
    if (!use_tol) {
        for (int iter = 0; iter < maxiter; ++iter) {
            IPTGB_CHECK(op.step(X[iter & 1], X[(iter + 1) & 1], d, 0, &scratch->ns));
        }
        IPTGB_CHECK(op.check());
        *X_final = X[maxiter & 1];
        *iterations_done = maxiter;
        *fixed_point_residual = NAN;
        return IPT_CUDA_SUCCESS;
    }
    // Tolerance mode: the host judges every step, and the GPU would wait ~25 us
    // for it (the norms' copy, the synchronisation and the next launches; a
    // step at n = 1024, k = 8 takes less).  So the next step is launched
    // before the norms of the running one are known, unless the residuals so
    // far say that the running step meets the tolerance.  A step past the
    // converged one writes only the block that step read.
    double *slots = pinned_norm_slots();
    if (slots == nullptr) return IPT_CUDA_ALLOCATION_FAILED;
    double *const device_norms = scratch->ns.norms;
    int launched = 0, status = IPT_CUDA_SUCCESS;
    double r1 = NAN, r2 = NAN;  // the last two residuals
    auto launch = [&]() -> int {
        double *slot = slots + 2 * (launched % kNormSlots);
        arm_slot(reinterpret_cast<volatile uint64_t *>(slot));
        scratch->ns.norms = slot;
        IPTGB_CHECK(op.step_ahead(X[launched & 1], X[(launched + 1) & 1], d, &scratch->ns));
        ++launched;
        return IPT_CUDA_SUCCESS;
    };
    int done = 0;
    while (done < maxiter) {
        if (launched == done) status = launch();
        const bool expect_stop = r1 * r1 <= 2.0 * tol * r2;
        if (status == IPT_CUDA_SUCCESS && launched == done + 1 && launched < maxiter &&
            !expect_stop) {
            status = launch();
        }
        const double *slot = slots + 2 * (done % kNormSlots);
        if (status == IPT_CUDA_SUCCESS && launched == done + 1) status = op.flush_norms();
        if (status == IPT_CUDA_SUCCESS) {
            status = wait_slot(reinterpret_cast<const volatile uint64_t *>(slot), stream);
        }
        if (status != IPT_CUDA_SUCCESS) break;
        const double delta_norm = slot[0];
        const double current_norm = slot[1];
        if (current_norm <= 0.0 || !isfinite(current_norm)) {
            status = IPT_CUDA_INVALID_ARGUMENT;
            break;
        }
        ++done;
        r2 = r1;
        r1 = delta_norm / current_norm;
        if (r1 <= tol) break;
    }
    // no step may still be writing a slot (or X) once this call returns
    if (status != IPT_CUDA_SUCCESS) {
        cudaStreamSynchronize(stream);
    } else if (launched > done) {
        status = op.flush_norms();
        if (status == IPT_CUDA_SUCCESS) {
            status = wait_slot(reinterpret_cast<const volatile uint64_t *>(
                                   slots + 2 * ((launched - 1) % kNormSlots)),
                               stream);
        }
    }
    scratch->ns.norms = device_norms;
    // (a step that failed leaves no finite norms)
    if (status == IPT_CUDA_INVALID_ARGUMENT) IPTGB_CHECK(op.check());
    IPTGB_CHECK(status);
    *X_final = X[done & 1];
    *iterations_done = done;
    *fixed_point_residual = r1;
    return IPT_CUDA_SUCCESS;
}

}  // namespace iptgb
