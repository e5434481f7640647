// reduce.cuh - deterministic block and grid reductions used by the kernels.
//
// Grid-wide sums use the "last block finishes" pattern: every block writes
// its partial to a slot indexed by blockIdx, the block that takes the final
// ticket sums the slots in a fixed order and resets the ticket counter.  The
// result therefore does not depend on block scheduling.
#pragma once

#include <cuda_runtime.h>

namespace iptgb {

// The sums below add pairs at distance 16, 8, 4, 2, 1, the same tree for each
// value.  An FP64 instruction holds its partition's pipe for 64 cycles whatever
// its lanes do, so the values share them: after the step at distance 16 the
// lower half of the warp carries on with a, the upper half with b.

// v at distance 16 (lower half: a, upper half: b).
__device__ __forceinline__ double pair_fold16(double a, double b)
{
    const bool up = (threadIdx.x & 16) != 0;
    const double got = __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
    return (up ? b : a) + got;
}

// Sum over the `nw` warps' values of slot lane / 16 (vals[slot][warp]) by one
// warp; lane 0 holds slot 0's, lane 16 slot 1's.
__device__ __forceinline__ double warps_fold(const double (*vals)[32], int nw)
{
    const int lane = threadIdx.x & 31;
    const double *v = vals[lane >> 4];
    const int i = lane & 15;
    double x = i < nw ? v[i] : 0.0;
    if (nw > 16) x += i + 16 < nw ? v[i + 16] : 0.0;
    for (int off = 8; off > 0; off >>= 1) {
        if (nw > off) x += __shfl_xor_sync(0xffffffffu, x, off);
    }
    return x;
}

// Block-wide sum of two doubles; the result is valid in thread 0.  Must be
// called by every thread of the block (it synchronises).
__device__ __forceinline__ double2 block_sum2(double a, double b)
{
    __shared__ double part[2][32];
    double x = pair_fold16(a, b);
    for (int off = 8; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    __syncthreads();
    if ((lane & 15) == 0) part[lane >> 4][warp] = x;
    __syncthreads();
    if (warp == 0) x = warps_fold(part, (blockDim.x + 31) >> 5);
    const double y = __shfl_down_sync(0xffffffffu, x, 16);
    __syncthreads();
    return make_double2(x, y);
}

// Two block_sum2 at once, for a block of at least two warps; ab and cd are
// valid in thread 0 (six FP64 additions per warp for four values, not twenty).
__device__ __forceinline__ void block_sum4(double2 &ab, double2 &cd)
{
    __shared__ double part[4][32];
    __shared__ double2 second;
    double x = pair_fold16(ab.x, ab.y);
    const double z = pair_fold16(cd.x, cd.y);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const bool up = (lane & 8) != 0;  // these lanes carry on with (c, d)
    const double got = __shfl_xor_sync(0xffffffffu, up ? x : z, 8);
    x = (up ? z : x) + got;
    for (int off = 4; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    __syncthreads();
    // lanes 0, 8, 16, 24: a, c, b, d
    if ((lane & 7) == 0) part[((lane >> 4) & 1) | ((lane >> 2) & 2)][warp] = x;
    __syncthreads();
    if (warp < 2) x = warps_fold(part + 2 * warp, (blockDim.x + 31) >> 5);
    const double y = __shfl_down_sync(0xffffffffu, x, 16);
    if (threadIdx.x == 32) second = make_double2(x, y);
    __syncthreads();
    ab = make_double2(x, y);
    cd = second;
}

// Warp-wide sum; every lane receives the total.
__device__ __forceinline__ double warp_sum(double v)
{
    for (int off = 16; off > 0; off >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, off);
    }
    return v;
}

// out[0] = sqrt(t.x), out[1] = sqrt(t.y) of a t valid in thread 0, by one warp
// (one square root's instructions for both).  Called by the whole block.
__device__ __forceinline__ void write_norms2(double2 t, double *out)
{
    if (threadIdx.x >= 32) return;
    const double y = __shfl_sync(0xffffffffu, t.y, 0);
    const double v = sqrt(threadIdx.x == 0 ? t.x : y);
    if (threadIdx.x < 2) out[threadIdx.x] = v;
}

// Deterministic grid-wide finish of per-block (a, b) sums.  `mine` must be
// valid in thread 0.  The last block writes out[0] = sqrt(sum a) and
// out[1] = sqrt(sum b) and re-arms *counter for the next launch.
__device__ __forceinline__ void grid_finish_norms2(double2 mine, double2 *partials,
                                                   unsigned int *counter, double *out)
{
    __shared__ bool last;
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = mine;
        __threadfence();
        const unsigned int done = atomicAdd(counter, 1u);
        last = (done == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) {
        return;
    }
    __threadfence();
    double a = 0.0, b = 0.0;
    for (unsigned int i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
        const double2 p = __ldcg(&partials[i]);
        a += p.x;
        b += p.y;
    }
    write_norms2(block_sum2(a, b), out);
    if (threadIdx.x == 0) *counter = 0u;
}

}  // namespace iptgb
