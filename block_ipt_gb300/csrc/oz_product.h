// oz_product.h - FP64-accurate dense block product on the tensor cores
// (internal; k_oz.cu, operand splitting in oz.cuh).
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernels.cuh"

namespace iptgb {

// The matrix of a product: an FP64 column-major n x n H in device memory
// (which must outlive the object's uses) and one exponent per row of
// Delta = H - diag(H).  With digit words the product streams those (8 bytes
// per entry, as H itself, but without the ~25 integer instructions per entry
// that the extraction of the digits takes in every product); without them it
// reads H and extracts the digits on the way.
struct OzMatrix {
    const double *H = nullptr;
    int n = 0;
    int nst = 0;           // 32-element K stages of a row
    int blocks = 0;        // kOzBlock-element blocks of a row
    int words_slices = 0;  // digits per entry in `words` (0: none)
    // settle() after build_words(7): entries of a row span more binades within
    // a block than the 56-bit split multiplies as accurately as FP64 FMAs
    // (oz_range_limit)
    bool wide = false;
    DeviceBuffer<int> rowexp;
    DeviceBuffer<uint16_t> blockexp;  // [block][row], oz_pack_exponent
    DeviceBuffer<uint4> words;  // oz_word_index
    OzMatrix() = default;
    ~OzMatrix();
    // H alone, for products in FP64 FMAs
    void reference(const double *H, int n);
    int init_storage(int n, cudaStream_t s);
    // storage of the words only (the mixed solve's fused setup writes them)
    int alloc_words(int slices, cudaStream_t s);
    // row exponents of H from one pass over it; diag (optional, n) receives
    // its diagonal
    int scan_rows(const double *H, int n, double *diag, cudaStream_t s);
    // digit words from a second pass (for matrices multiplied more than once
    // or twice); without an error none where they exceed kMaxWordMb or the
    // device's memory.  slices = 7: also finds out whether the matrix is
    // `wide`, which settle() waits for; a wide one then has no words.
    // Until the object goes, an allocation of this thread that fails takes the
    // words' memory (reclaim_memory): the products then read H.
    int build_words(int slices, cudaStream_t s);
    int settle(cudaStream_t s);
    bool drop_words(cudaStream_t s);
    int *answer = nullptr;        // page-locked, while settle() is due
    OzMatrix *held_before = nullptr;  // the thread's list of matrices with words
    bool listed = false;
};

// The most memory the words may take, MB (n up to 46340); they go back to the
// stream-ordered pool after a solve.  Tuning and test knob IPT_GB300_WORDS_MAX_MB
// (0: the product always extracts the digits itself).
constexpr int kMaxWordMb = 16384;

// Launch shape of a product with C columns: `groups` column groups of cp
// columns; the work items (group, 128-row tile, period of K elements) are
// split evenly over `grid` persistent CTAs.
struct OzShape {
    int n = 0, C = 0, cp = 0, groups = 0, tiles = 0, periods = 0, ldp = 0, grid = 0;
    int spp = 0;       // 32-element K stages per item
    int maxslots = 0;  // partials a (group, tile) can have; FP64 FMAs: K slices
    long long items = 0;
};

// Y = (diag(d) + Delta) X for an n x C block X (column-major, ld ldx); d may
// be null (Y = Delta X).  slices = 6: the 48-bit split; 7: the 56-bit split
// of the plain FP64 path (oz.cuh), for matrices that are not `wide`; 0: no split, FP64 FMAs (k_dense64.cu; step()
// only).
namespace oz {
struct Partials;
}
struct OzProduct {
    const OzMatrix *m = nullptr;
    const double *d = nullptr;
    cudaStream_t s = nullptr;
    int sms = 148;
    int slices = 6;
    OzShape sh;
    DeviceBuffer<__half> B;
    DeviceBuffer<int> colexp;
    DeviceBuffer<uint16_t> xexp;  // slices = 7: [group][block][cp], oz_pack_exponent
    DeviceBuffer<unsigned long long> colmax;  // two sets of C column maxima
    int cur = 0;                              // the set the next product reads
    // deferred norms of the last step: parts, their number (0: none), target
    const double2 *pending_parts = nullptr;
    int pending_count = 0;
    double *pending_out = nullptr;
    DeviceBuffer<double> P;
    DeviceBuffer<int> err;
    CUtensorMap mapB;
    int bind(const OzMatrix *matrix, const double *diag, int digit_slices, cudaStream_t stream);
    int apply(const double *X, long long ldx, int C, double *Y, long long ldy);

    // The plain IPT loop keeps the column maxima of its iterate up to date
    // itself: begin() scans the first block, step() forms Delta X from the
    // maxima of set `cur` and then Xn = F(X) (IPT map with g = 1 / (d_j - d_i),
    // n x C; null: the ACX map, which divides), the maxima of Xn in the other set, and with ns (want_norms)
    // ||Xn - X||_F and ||X||_F in ns->norms.
    int begin(const double *X, int C);
    // resid_part (optional): update_row_blocks parts per column of
    // ||(H X)_c - X_c (H X)_cc||^2.
    // defer_norms: the norms reach ns->norms with the next step, or with
    // flush_norms() where none follows.
    int step(const double *X, const double *g, double *Xn, int want_norms, NormScratch *ns,
             double *resid_part = nullptr, bool defer_norms = false);
    int flush_norms();
    static int update_row_blocks(int n, int C, int sms, bool *wide);
    // the column maxima (bit patterns) the next step reads
    // (null with FP64 FMAs)
    unsigned long long *column_maxima()
    {
        return slices == 0 ? nullptr : colmax.ptr + (size_t)cur * sh.groups * sh.cp;
    }

    // polls of a pipeline wait before the kernel gives up (tuning and test knob
    // IPT_GB300_SPIN_LIMIT; the drain before TMEM is released always uses the
    // full bound)
    long long spin = 0;
    // the kernel's error flag (non-zero: a bounded wait gave up); waits for the
    // stream
    int read_error(int *host_err);
    // IPT_CUDA_CUDA_ERROR where it is set, as the results are then NaN
    int check();

  private:
    int shape_for(int C);
    int scan_columns(const double *X, long long ldx);
    int slice_and_multiply(const double *X, long long ldx, int clear_other);
    oz::Partials partials() const;
};

// Does the caller's environment ask for FP64 FMAs (IPT_GB300_FP64_DFMA=1 or
// IPT_GB300_ACCURATE_PRODUCT=fp64)?
bool fp64_fma_wanted();

// g_ij = 1 / (d_j - d_i) for the n x k block (NaN for a zero or non-finite
// gap, as the reference's build_g_kernel with min_gap_allowed = 0).
int launch_gap_reciprocals(const double *d, int n, int k, double *g, cudaStream_t s);

}  // namespace iptgb
