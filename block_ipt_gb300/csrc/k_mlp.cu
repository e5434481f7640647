// k_mlp.cu - learned Davidson preconditioner: a per-row MLP (6 -> 64 -> 64
// -> 1, ReLU) that replaces the plain diagonal correction
// t_i = r_i / (d_i - theta) of the reference's Davidson step
// (IPT_C_GPU/src/ipt_cuda.cu:2449-2465, clip rule :3389-3403).
//
// The exact correction of a Ritz pair (theta, x, r) is (H - theta)^-1 r; with
// H = D + Delta its Neumann series starts t1 + u with the plain correction
// t1 = (D - theta)^-1 r and the second-order term u = -(D - theta)^-1 Delta t1,
// which costs one product with H (H t1, the diagonal part taken off).  The
// learned correction is t_i = t1_i + o_i u_i with the network's per-row
// weight o_i = sigmoid(z_i), z_i its linear output: o -> 1 everywhere is the
// two-term Neumann correction, near which training starts (output bias 4:
// o = 0.982), o -> 0 the plain preconditioner.  The two-term correction is
// a strong baseline on the FCI-like family (it saves about 40 % of the
// Davidson steps of the plain one); the network learns per row how much of
// the second-order term to keep, never more than all of it.  Features of
// row i, all O(1):
//   f0 = t1_i sqrt(n) / ||t1||       plain correction, normalised
//   f1 = u_i sqrt(n) / ||t1||        second-order term, same units
//   f2 = x_i sqrt(n)                 Ritz vector (unit norm)
//   f3 = asinh((d_i - theta) / s_i)  gap in units of the row's off-diagonal
//                                    coupling s_i = ||H[i, j != i]||_2
//   f4 = asinh(s_i / (|d_i - theta| + clip))
//   f5 = log10(||r|| / max(1, ||H||_inf)) / 8   convergence level
//
// Training target (what the collector records while the plain solver runs
// against the converged eigenvectors x*): the part of the exact error that
// lies outside the current search space V, e = (I - V V^T)(s x*_l - x)
// (x*_l the converged vector that overlaps x most, s its sign), scaled by
// the least-squares fit e ~ alpha (I - V V^T)(t1 + u).  Davidson keeps only
// the part of a correction outside V, so the targets compare projected
// vectors: with p = (I - V V^T) t1 and q = (I - V V^T) u, per row the weight
// that reproduces the scaled error, y_i = (e_i / alpha - p_i) / q_i, with
// weight w_i = n q_i^2 / ||t1||^2, so that the weighted loss
// sum_i w_i (o_i - y_i)^2 equals ||p + o o q - e / alpha||^2 in the units
// of f1: for o = 1 (the two-term correction) and o = 0 (the plain one) it is
// the error of exactly the direction the Davidson step adds.  (Comparing the
// unprojected t1 + o u instead ranks the two-term correction below the plain
// one, although it saves Davidson steps: its components inside V count
// against it there and are discarded by the step.)
//
// Training runs on the GPU: a fused forward/backward kernel over row tiles of
// a batch (per-tile gradient partials, no atomics) and an Adam kernel that sums
// the partials in a fixed order, so a training run is deterministic for a
// given seed.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "block_ops.h"
#include "block_solver.h"
#include "common.cuh"
#include "ipt_plain.h"
#include "reduce.cuh"

namespace iptgb {
namespace mlp {

constexpr int kIn = 6;
constexpr int kH = 64;
constexpr int kRow = kIn + 2;  // features, target, weight
constexpr int oW1 = 0;
constexpr int oB1 = oW1 + kH * kIn;
constexpr int oW2 = oB1 + kH;
constexpr int oB2 = oW2 + kH * kH;
constexpr int oW3 = oB2 + kH;
constexpr int oB3 = oW3 + kH;
constexpr int kParams = oB3 + 1;  // 4673

__host__ __device__ constexpr int param_count() { return kParams; }

__device__ __forceinline__ unsigned long long splitmix(unsigned long long x)
{
    x += 0x9E3779B97F4A7C15ULL;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
    return x ^ (x >> 31);
}

__device__ __forceinline__ float clampf(float v, float lim)
{
    if (!(v == v)) return 0.f;  // NaN
    return fminf(fmaxf(v, -lim), lim);
}


__device__ __forceinline__ void row_features(double t, double tn, double u, double rn, double x,
                                             double delta, double sigma, double clip,
                                             double hnorm, int n, float f[kIn])
{
    const double sn = sqrt((double)n);
    f[0] = clampf((float)(tn > 0.0 ? t * sn / tn : 0.0), 40.f);
    f[1] = clampf((float)(tn > 0.0 ? u * sn / tn : 0.0), 40.f);
    f[2] = clampf((float)(x * sn), 40.f);
    const double s = sigma + 1e-12 * fmax(1.0, fabs(hnorm));
    f[3] = clampf((float)asinh(delta / s), 40.f);
    f[4] = clampf((float)asinh(sigma / (fabs(delta) + clip)), 40.f);
    f[5] = clampf((float)(log10(rn / fmax(1.0, hnorm) + 1e-300) / 8.0), 40.f);
}

// Weight of the second-order term from the network's linear output z.
constexpr float kOutBias = 4.f;  // initial z: o = sigmoid(4) = 0.982
__device__ __forceinline__ float weight_of(float z) { return 1.f / (1.f + expf(-z)); }

// o = sigmoid(z), z = W3 relu(W2 relu(W1 f + b1) + b2) + b3, with the
// parameters in shared memory
__device__ __forceinline__ float forward_row(const float *__restrict__ P, const float f[kIn])
{
    float h1[kH];
#pragma unroll
    for (int j = 0; j < kH; ++j) {
        float s = P[oB1 + j];
#pragma unroll
        for (int q = 0; q < kIn; ++q) s = fmaf(P[oW1 + j * kIn + q], f[q], s);
        h1[j] = fmaxf(s, 0.f);
    }
    float o = P[oB3];
    for (int j = 0; j < kH; ++j) {
        const float4 *w = reinterpret_cast<const float4 *>(P + oW2 + j * kH);
        float s = P[oB2 + j];
#pragma unroll
        for (int l4 = 0; l4 < kH / 4; ++l4) {
            const float4 ww = w[l4];
            s = fmaf(ww.x, h1[4 * l4 + 0], s);
            s = fmaf(ww.y, h1[4 * l4 + 1], s);
            s = fmaf(ww.z, h1[4 * l4 + 2], s);
            s = fmaf(ww.w, h1[4 * l4 + 3], s);
        }
        o = fmaf(P[oW3 + j], fmaxf(s, 0.f), o);
    }
    return weight_of(o);
}

__device__ __forceinline__ void load_params(const float *__restrict__ g, float *s)
{
    for (int p = threadIdx.x; p < kParams; p += blockDim.x) s[p] = g[p];
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Initialisation: weights U(-a, a) with a = sqrt(6 / fan_in) (ReLU layers) and
// 0.1 sqrt(3 / fan_in) (linear output), hidden biases 0, output bias
// kOutBias (so o starts near 1, the two-term correction); counter-based,
// seeded.
// ---------------------------------------------------------------------------
__global__ void mlp_init_kernel(float *__restrict__ params, unsigned long long seed)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kParams) return;
    float a = 0.f;
    if (p < oB1) a = sqrtf(6.f / kIn);
    else if (p >= oW2 && p < oB2) a = sqrtf(6.f / kH);
    else if (p >= oW3 && p < oB3) a = 0.1f * sqrtf(3.f / kH);
    const unsigned long long h = splitmix(seed * 0x100000001B3ULL + (unsigned long long)p);
    const float u = (float)((h >> 11) * (1.0 / 9007199254740992.0));  // [0, 1)
    params[p] = p == oB3 ? kOutBias : a * (2.f * u - 1.f);
}

// ---------------------------------------------------------------------------
// Inference on stored feature rows (row stride `ld` floats): out[r] = MLP(f).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
mlp_forward_rows_kernel(const float *__restrict__ params, const float *__restrict__ rows,
                        long long nrows, int ld, float *__restrict__ out)
{
    __shared__ __align__(16) float P[kParams + 3];
    load_params(params, P);
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    float f[kIn];
#pragma unroll
    for (int q = 0; q < kIn; ++q) f[q] = rows[r * ld + q];
    out[r] = forward_row(P, f);
}

// ---------------------------------------------------------------------------
// Fused forward + backward over a batch.  Loss: mean over the batch of
// w (o - y)^2 with o = sigmoid(z) (row = f0..f5, y, w).  Row b of the batch is
// row b of `rows` (sample = 0) or a seeded hash of (seed, step, b) modulo
// nrows (sample = 1).  partials[tile][p] = d loss / d param_p restricted to the
// tile, and partials[tile][kParams] = its sum of weighted squared errors.
//
// A CTA of 256 threads takes tiles of 128 rows, one after the other (the
// weights stay in shared memory).  The three 64 x 64 products of a row (W2 h1,
// W2^T d2, d2 h1^T) are register-tiled FP32 products of shared-memory
// operands: 8 x 4 outputs per thread, 16-byte reads along K for the rows (the
// two row groups of a warp in different banks, ld = 68) and of 4 columns, 128
// FMAs per 12 reads.  Every sum runs in the order of its index (units, then
// the rows of the tile), one thread per sum, so the bits of a gradient - and
// of a training run, whose course is sensitive to them - do not depend on the
// launch shape.
//
// Bound by the FP32 pipe and the reads beside it (3 x 4096 FMAs per row: 66
// us at 200,000 rows).  One row per thread with scalar shared-memory reads of
// one weight per FMA took 635 us there, and 180 us for a single tile;
// now 193 us and 24 us, the sum over the tiles 15 us instead of 66 us.
// ---------------------------------------------------------------------------
constexpr int kTile = 128;       // rows of a tile
constexpr int kFbThreads = 256;
constexpr int kLd = kH + 4;

struct FbShared {
    float W2t[kH][kH];       // [l][j]
    float W2[kH][kH];        // [j][l]
    float W1[kH][8];         // 6 weights, bias, pad
    float b2[kH], W3[kH];
    float H1[kTile][kLd], H2[kTile][kLd], D1[kTile][kLd], D2[kTile][kLd];
    float F[kTile][kRow];
    float G[kTile];          // d loss / d z of the tile's rows
    float sq[kTile];         // weighted squared errors
};

constexpr int kTR = kTile / 16;  // rows per thread

// acc[i][c] += sum_k A[rg + 16 i][k] B[k][4 cg + c], k ascending
__device__ __forceinline__ void tile_product(const float (*__restrict__ A)[kLd],
                                             const float (*__restrict__ B)[kH], int rg, int cg,
                                             float (&acc)[kTR][4])
{
#pragma unroll 2
    for (int k = 0; k < kH; k += 4) {
        float4 b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = *reinterpret_cast<const float4 *>(&B[k + u][4 * cg]);
#pragma unroll
        for (int i = 0; i < kTR; ++i) {
            const float4 av = *reinterpret_cast<const float4 *>(&A[rg + 16 * i][k]);
            const float a[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                acc[i][0] = fmaf(a[u], b[u].x, acc[i][0]);
                acc[i][1] = fmaf(a[u], b[u].y, acc[i][1]);
                acc[i][2] = fmaf(a[u], b[u].z, acc[i][2]);
                acc[i][3] = fmaf(a[u], b[u].w, acc[i][3]);
            }
        }
    }
}

__global__ void __launch_bounds__(kFbThreads, 1)
mlp_fwd_bwd_kernel(const float *__restrict__ params, const float *__restrict__ rows,
                   long long nrows, int batch, int tiles, int sample, unsigned long long seed,
                   int step, float *__restrict__ partials)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    FbShared &S = *reinterpret_cast<FbShared *>(sm_raw);
    const int t = threadIdx.x;
    const int cg = t & 15, rg = t >> 4;
    for (int e = t; e < kH * kH; e += kFbThreads) {
        const float w = params[oW2 + e];
        S.W2[e / kH][e % kH] = w;
        S.W2t[e % kH][e / kH] = w;
    }
    for (int e = t; e < kH * kIn; e += kFbThreads) S.W1[e / kIn][e % kIn] = params[oW1 + e];
    if (t < kH) {
        S.W1[t][6] = params[oB1 + t];
        S.W1[t][7] = 0.f;
        S.b2[t] = params[oB2 + t];
        S.W3[t] = params[oW3 + t];
    }
    const float bias3 = params[oB3];
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();  // the previous tile's operands have been read
        for (int e = t; e < kTile * kRow; e += kFbThreads) {
            const int i = e / kRow;
            const int b = tile * kTile + i;
            float v = 0.f;
            if (b < batch) {
                long long r = b;
                if (sample) {
                    const unsigned long long h = splitmix(
                        seed ^ ((unsigned long long)step << 32) ^ (unsigned long long)b);
                    r = (long long)(h % (unsigned long long)nrows);
                }
                v = rows[r * kRow + e % kRow];
            }
            S.F[i][e % kRow] = v;
        }
        __syncthreads();
        // layer 1
#pragma unroll
        for (int i = 0; i < kTR; ++i) {
            const float *f = S.F[rg + 16 * i];
            float h[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float *w = S.W1[4 * cg + c];
                float v = w[6];
#pragma unroll
                for (int q = 0; q < kIn; ++q) v = fmaf(w[q], f[q], v);
                h[c] = fmaxf(v, 0.f);
            }
            *reinterpret_cast<float4 *>(&S.H1[rg + 16 * i][4 * cg]) =
                make_float4(h[0], h[1], h[2], h[3]);
        }
        __syncthreads();
        // layer 2
        float acc[kTR][4];
#pragma unroll
        for (int i = 0; i < kTR; ++i) {
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][c] = S.b2[4 * cg + c];
        }
        tile_product(S.H1, S.W2t, rg, cg, acc);
#pragma unroll
        for (int i = 0; i < kTR; ++i) {
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][c] = fmaxf(acc[i][c], 0.f);
            *reinterpret_cast<float4 *>(&S.H2[rg + 16 * i][4 * cg]) =
                make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        __syncthreads();
        // output and its gradient, one row per thread
        if (t < kTile) {
            float z = bias3;
#pragma unroll
            for (int j = 0; j < kH; j += 4) {
                const float4 h = *reinterpret_cast<const float4 *>(&S.H2[t][j]);
                z = fmaf(S.W3[j + 0], h.x, z);
                z = fmaf(S.W3[j + 1], h.y, z);
                z = fmaf(S.W3[j + 2], h.z, z);
                z = fmaf(S.W3[j + 3], h.w, z);
            }
            const float sg = weight_of(z);
            const bool valid = tile * kTile + t < batch;
            const float y = S.F[t][kIn], wgt = S.F[t][kIn + 1];
            const float err = valid ? sg - y : 0.f;
            // d loss / d z through o = sigmoid(z)
            S.G[t] = valid ? 2.f * wgt * err * sg * (1.f - sg) / (float)batch : 0.f;
            S.sq[t] = wgt * err * err;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kTR; ++i) {
            const float g = S.G[rg + 16 * i];
            float d2[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) d2[c] = acc[i][c] > 0.f ? S.W3[4 * cg + c] * g : 0.f;
            *reinterpret_cast<float4 *>(&S.D2[rg + 16 * i][4 * cg]) =
                make_float4(d2[0], d2[1], d2[2], d2[3]);
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
        }
        __syncthreads();
        // back through layer 2
        tile_product(S.D2, S.W2, rg, cg, acc);
#pragma unroll
        for (int i = 0; i < kTR; ++i) {
            const float4 h = *reinterpret_cast<const float4 *>(&S.H1[rg + 16 * i][4 * cg]);
            *reinterpret_cast<float4 *>(&S.D1[rg + 16 * i][4 * cg]) =
                make_float4(h.x > 0.f ? acc[i][0] : 0.f, h.y > 0.f ? acc[i][1] : 0.f,
                            h.z > 0.f ? acc[i][2] : 0.f, h.w > 0.f ? acc[i][3] : 0.f);
        }
        __syncthreads();
        // gradients of the tile, rows ascending
        float *out = partials + (size_t)tile * (kParams + 1);
        {
            // dW2[j][l] = sum over rows of d2 h1, 4 x 4 per thread
            const int jg = rg;
            float w[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int c = 0; c < 4; ++c) w[j][c] = 0.f;
            }
#pragma unroll 8
            for (int r = 0; r < kTile; ++r) {
                const float4 h = *reinterpret_cast<const float4 *>(&S.H1[r][4 * cg]);
                const float4 u = *reinterpret_cast<const float4 *>(&S.D2[r][4 * jg]);
                const float dj[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    w[j][0] = fmaf(dj[j], h.x, w[j][0]);
                    w[j][1] = fmaf(dj[j], h.y, w[j][1]);
                    w[j][2] = fmaf(dj[j], h.z, w[j][2]);
                    w[j][3] = fmaf(dj[j], h.w, w[j][3]);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    out[oW2 + (4 * jg + j) * kH + 4 * cg + c] = w[j][c];
                }
            }
        }
        // thread groups of 64: two columns of dW1 each, then the biases and W3
        const int j = t & 63;
        if (t < 192) {
            const int q = 2 * (t >> 6);
            float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
            for (int r = 0; r < kTile; ++r) {
                const float d = S.D1[r][j];
                s0 = fmaf(d, S.F[r][q], s0);
                s1 = fmaf(d, S.F[r][q + 1], s1);
            }
            out[oW1 + j * kIn + q] = s0;
            out[oW1 + j * kIn + q + 1] = s1;
        } else {
            float s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 8
            for (int r = 0; r < kTile; ++r) {
                s1 += S.D1[r][j];
                s2 += S.D2[r][j];
                s3 = fmaf(S.G[r], S.H2[r][j], s3);
            }
            out[oB1 + j] = s1;
            out[oB2 + j] = s2;
            out[oW3 + j] = s3;
        }
        if (t == 0 || t == 64) {
            const float *v = t == 0 ? S.G : S.sq;
            float s = 0.f;
#pragma unroll 8
            for (int r = 0; r < kTile; ++r) s += v[r];
            out[t == 0 ? oB3 : kParams] = s;
        }
    }
}

int fb_tiles(int batch) { return (batch + kTile - 1) / kTile; }

int launch_fwd_bwd(const float *params, const float *rows, long long nrows, int batch, int sample,
                   unsigned long long seed, int step, float *partials, cudaStream_t s)
{
    const int tiles = fb_tiles(batch);
    const int ctas = std::min(tiles, device_sm_count());
    const size_t smem = sizeof(FbShared);
    IPTGB_CUDA(cudaFuncSetAttribute(mlp_fwd_bwd_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    mlp_fwd_bwd_kernel<<<ctas, kFbThreads, smem, s>>>(params, rows, nrows, batch, tiles, sample,
                                                      seed, step, partials);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

// Sums of 32 parameters p0 + lane over the tiles, in tile order, valid in the
// threads of warp 0 of a 256-thread block.  The adds of a parameter are one
// chain; the eight warps bring 128 tiles' values into shared memory while
// warp 0 adds the previous 128 (one thread per parameter reading global
// memory itself waits out a load latency every few adds: 51 us for the 1563
// tiles of 200,000 rows).
constexpr int kSumThreads = 256;
constexpr int kSumChunk = 128;

__device__ __forceinline__ float sum_tiles(const float *__restrict__ partials, int tiles, int p0)
{
    __shared__ float buf[2][kSumChunk][32];
    constexpr int kPer = kSumChunk / (kSumThreads / 32);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool live = p0 + lane <= kParams;
    auto load = [&](int c, float (&v)[kPer]) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int b = c * kSumChunk + warp * kPer + u;
            v[u] = live && b < tiles ? partials[(size_t)b * (kParams + 1) + p0 + lane] : 0.f;
        }
    };
    const int chunks = (tiles + kSumChunk - 1) / kSumChunk;
    float v[kPer];
    load(0, v);
    float s = 0.f;
    for (int c = 0; c < chunks; ++c) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) buf[c & 1][warp * kPer + u][lane] = v[u];
        if (c + 1 < chunks) load(c + 1, v);
        __syncthreads();
        if (warp == 0) {
            const int count = min(kSumChunk, tiles - c * kSumChunk);
#pragma unroll 16
            for (int u = 0; u < count; ++u) s += buf[c & 1][u][lane];
        }
    }
    return s;
}

// Sum of the tile partials in tile order: grad[p] (p < kParams) and
// grad[kParams] = the batch loss.
__global__ void __launch_bounds__(kSumThreads)
mlp_grad_finish_kernel(const float *__restrict__ partials, int tiles, int batch,
                       float *__restrict__ grad)
{
    const float s = sum_tiles(partials, tiles, blockIdx.x * 32);
    const int p = blockIdx.x * 32 + threadIdx.x;
    if (threadIdx.x >= 32 || p > kParams) return;
    grad[p] = p == kParams ? s / (float)batch : s;
}

// Adam (Kingma & Ba 2015): m = b1 m + (1-b1) g, v = b2 v + (1-b2) g^2,
// p -= lr m_hat / (sqrt(v_hat) + eps); step is 1-based.
__global__ void __launch_bounds__(kSumThreads)
mlp_adam_kernel(float *__restrict__ params, float *__restrict__ m,
                                float *__restrict__ v, const float *__restrict__ partials,
                                int tiles, int batch, int step, float lr,
                                float *__restrict__ loss_hist)
{
    const float g = sum_tiles(partials, tiles, blockIdx.x * 32);
    const int p = blockIdx.x * 32 + threadIdx.x;
    if (threadIdx.x >= 32 || p > kParams) return;
    if (p == kParams) {
        if (loss_hist != nullptr) loss_hist[step - 1] = g / (float)batch;
        return;
    }
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mm = b1 * m[p] + (1.f - b1) * g;
    const float vv = b2 * v[p] + (1.f - b2) * g * g;
    m[p] = mm;
    v[p] = vv;
    const float mh = mm / (1.f - powf(b1, (float)step));
    const float vh = vv / (1.f - powf(b2, (float)step));
    params[p] -= lr * mh / (sqrtf(vh) + eps);
}

// ---------------------------------------------------------------------------
// Davidson use.  second_order_kernel turns U = H t1 into the second-order
// term u = -(D - theta)^-1 (H t1 - D t1) (denominators clipped like the plain
// correction); mlp_correct_kernel computes the features of every (row,
// selected pair), runs the MLP and leaves t1 + clamp(o) u in T.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double clipped_gap(double d, double theta, double clip)
{
    double den = d - theta;
    if (fabs(den) < clip) den = den < 0.0 ? -clip : clip;
    return den;
}

__global__ void second_order_kernel(const double *__restrict__ T, const double *__restrict__ d,
                                    const double *__restrict__ theta, const int *__restrict__ sel,
                                    int nsel, int n, double clip, double *__restrict__ U)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * nsel) return;
    const int i = (int)(idx % (size_t)n);
    const int c = (int)(idx / (size_t)n);
    const double den = clipped_gap(d[i], theta[sel[c]], clip);
    U[idx] = -(U[idx] - d[i] * T[idx]) / den;
}

__global__ void __launch_bounds__(256)
mlp_correct_kernel(const float *__restrict__ params, const double *__restrict__ U,
                   const double *__restrict__ X, const double *__restrict__ d,
                   const double *__restrict__ theta, const int *__restrict__ sel, int nsel,
                   int n, double clip, double hnorm, const double *__restrict__ sigma,
                   const double *__restrict__ tnorm, const double *__restrict__ rnorm,
                   double *__restrict__ T)
{
    __shared__ __align__(16) float P[kParams + 3];
    load_params(params, P);
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * nsel) return;
    const int i = (int)(idx % (size_t)n);
    const int c = (int)(idx / (size_t)n);
    const int j = sel[c];
    float f[kIn];
    const double u = U[idx];
    row_features(T[idx], tnorm[c], u, rnorm[j], X[(size_t)i + (size_t)j * n], d[i] - theta[j],
                 sigma[i], clip, hnorm, n, f);
    const float o = forward_row(P, f);
    T[idx] = fma((double)o, u, T[idx]);
}

__global__ void add_kernel(double *__restrict__ A, const double *__restrict__ B, size_t count)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < count) A[e] += B[e];
}

// Collector: E[:, c] = s_c Xstar[:, l_c] - X[:, sel_c] (n x nsel).
__global__ void collect_error_kernel(const double *__restrict__ Xstar, const int *__restrict__ lidx,
                                     const double *__restrict__ sgn, const double *__restrict__ X,
                                     const int *__restrict__ sel, int nsel, int n,
                                     double *__restrict__ E)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * nsel) return;
    const int i = (int)(idx % (size_t)n);
    const int c = (int)(idx / (size_t)n);
    E[idx] = sgn[c] * Xstar[(size_t)lidx[c] * n + i] - X[(size_t)i + (size_t)sel[c] * n];
}

// Collector pass 1: per selected pair c: dots[3c] = <E_c, T_c>,
// dots[3c+1] = <T_c, T_c>, dots[3c+2] = <E_c, E_c> (T: the projected
// two-term correction).
__global__ void collect_dots_kernel(const double *__restrict__ E, const double *__restrict__ T,
                                    int n, double *__restrict__ dots)
{
    const int c = blockIdx.x;
    const double *ec = E + (size_t)c * n;
    const double *t = T + (size_t)c * n;
    double et = 0.0, tt = 0.0, ee = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double e = ec[i];
        et = fma(e, t[i], et);
        tt = fma(t[i], t[i], tt);
        ee = fma(e, e, ee);
    }
    const double2 a = block_sum2(et, tt);
    const double2 b = block_sum2(ee, 0.0);
    if (threadIdx.x == 0) {
        dots[3 * c] = a.x;
        dots[3 * c + 1] = a.y;
        dots[3 * c + 2] = b.x;
    }
}

// Collector pass 2: rows (f0..f5, target scale, weight) of the valid pairs;
// slot[c] >= 0 is the pair's first row in `out`, alpha[c] the fit of E by T_c.
// Collector pass 2: rows (f0..f5, target weight, row weight) of the valid
// pairs; slot[c] >= 0 is the pair's first row in `out`, alpha[c] the fit of
// E by the projected two-term correction.
__global__ void collect_rows_kernel(const double *__restrict__ E, const double *__restrict__ alpha,
                                    const long long *__restrict__ slot,
                                    const double *__restrict__ U, const double *__restrict__ X,
                                    const double *__restrict__ d, const double *__restrict__ theta,
                                    const int *__restrict__ sel, int nsel, int n, double clip,
                                    double hnorm, const double *__restrict__ sigma,
                                    const double *__restrict__ tnorm,
                                    const double *__restrict__ rnorm, const double *__restrict__ T,
                                    const double *__restrict__ Tp, const double *__restrict__ Up,
                                    float *__restrict__ out)
{
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * nsel) return;
    const int i = (int)(idx % (size_t)n);
    const int c = (int)(idx / (size_t)n);
    if (slot[c] < 0) return;
    const int j = sel[c];
    const double tn = tnorm[c];
    float f[kIn];
    const double x = X[(size_t)i + (size_t)j * n];
    const double u = U[idx];
    row_features(T[idx], tn, u, rnorm[j], x, d[i] - theta[j], sigma[i], clip, hnorm, n, f);
    // the per-row weight of the projected u that reproduces the scaled exact
    // error with the projected t1; rows where it vanishes carry (almost) no
    // weight
    const double up = Up[idx];
    const double y = fabs(up) > 0.0 ? (E[idx] / alpha[c] - Tp[idx]) / up : 1.0;
    const float g = tn > 0.0 ? (float)(up * sqrt((double)n) / tn) : 0.f;
    float *o = out + (size_t)(slot[c] + i) * kRow;
#pragma unroll
    for (int q = 0; q < kIn; ++q) o[q] = f[q];
    o[kIn] = clampf((float)y, 5.f);
    o[kIn + 1] = g * g;
}

// Row coupling s_i = ||H[i, j != i]||_2 of a CSR matrix (one warp per row).
__global__ void csr_offdiag_norm_kernel(const int *__restrict__ row_ptr,
                                        const int *__restrict__ col_ind,
                                        const double *__restrict__ vals, int n,
                                        double *__restrict__ sigma)
{
    const int row = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    double s = 0.0;
    for (int p = row_ptr[row] + lane; p < row_ptr[row + 1]; p += 32) {
        const double v = col_ind[p] == row ? 0.0 : vals[p];
        s = fma(v, v, s);
    }
    s = warp_sum(s);
    if (lane == 0) sigma[row] = sqrt(s);
}

// Same for a dense symmetric column-major H (column i = row i; one CTA per row).
__global__ void dense_offdiag_norm_kernel(const double *__restrict__ H, int n,
                                          double *__restrict__ sigma)
{
    const int row = blockIdx.x;
    const double *col = H + (size_t)row * n;
    double s = 0.0;
    for (int l = threadIdx.x; l < n; l += blockDim.x) {
        const double v = l == row ? 0.0 : col[l];
        s = fma(v, v, s);
    }
    const double2 t = block_sum2(s, 0.0);
    if (threadIdx.x == 0) sigma[row] = sqrt(t.x);
}

}  // namespace mlp

int launch_csr_row_coupling(const int *row_ptr, const int *col_ind, const double *vals, int n,
                            double *sigma, cudaStream_t s)
{
    mlp::csr_offdiag_norm_kernel<<<blocks_for((size_t)n * 32), kThreads, 0, s>>>(row_ptr, col_ind,
                                                                                 vals, n, sigma);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

int launch_dense_row_coupling(const double *H, int n, double *sigma, cudaStream_t s)
{
    mlp::dense_offdiag_norm_kernel<<<n, 256, 0, s>>>(H, n, sigma);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

// T <- (I - V V^T) T for the n x nsel correction block (one pass; the solver
// re-orthogonalises every correction against V afterwards anyway).
static int project_out(BlockOps &ops, const CorrectionArgs &a, double *T, DeviceBuffer<double> &G)
{
    if (a.V == nullptr || a.m <= 0) return IPT_CUDA_SUCCESS;
    if (G.count < (size_t)a.m * a.nsel) IPTGB_CHECK(G.alloc((size_t)a.m * a.nsel, ops.stream));
    IPTGB_CHECK(ops.gram(a.V, a.n, a.m, T, a.n, a.nsel, a.n, G.ptr, a.m));
    return ops.tall_gemm(a.V, a.n, G.ptr, a.m, T, a.n, a.n, a.m, a.nsel, -1.0, 1.0);
}

// t1 (plain correction, in T) and the second-order term u (in U) of the
// selected pairs; tn = ||t1|| per pair.
static int plain_and_second_order(BlockOps &ops, const CorrectionArgs &a, double *T,
                                  DeviceBuffer<double> &U, double *tn)
{
    cudaStream_t s = ops.stream;
    const size_t nc = (size_t)a.n * a.nsel;
    IPTGB_CHECK(ops.diag_correction(a.R, a.d, a.theta, a.sel, a.nsel, a.n, a.clip, T));
    if (U.count < nc) IPTGB_CHECK(U.alloc(nc, s));
    if (a.apply == nullptr) return IPT_CUDA_INVALID_ARGUMENT;
    IPTGB_CHECK(a.apply->apply(T, a.nsel, U.ptr));
    mlp::second_order_kernel<<<blocks_for(nc), kThreads, 0, s>>>(T, a.d, a.theta, a.sel, a.nsel,
                                                                 a.n, a.clip, U.ptr);
    IPTGB_LAUNCH();
    return ops.column_norms(T, a.n, a.n, a.nsel, tn);
}

namespace {

// The learned correction used by the Davidson driver.
struct MlpCorrection final : LearnedCorrection {
    const float *params = nullptr;
    const double *sigma = nullptr;
    double hnorm = 1.0;
    BlockOps ops;
    DeviceBuffer<double> tn, U;
    void bind(const double *row_coupling, double h) override
    {
        sigma = row_coupling;
        hnorm = h;
    }
    bool learned() const override { return true; }
    int correct(const CorrectionArgs &a, double *T) override
    {
        KernelTimerScope timer(kProfMlp, ops.stream);
        if (tn.count < (size_t)a.nsel) IPTGB_CHECK(tn.alloc((size_t)a.nsel, ops.stream));
        IPTGB_CHECK(plain_and_second_order(ops, a, T, U, tn.ptr));
        mlp::mlp_correct_kernel<<<blocks_for((size_t)a.n * a.nsel), 256, 0, ops.stream>>>(
            params, U.ptr, a.X, a.d, a.theta, a.sel, a.nsel, a.n, a.clip, hnorm, sigma, tn.ptr,
            a.rnorm, T);
        IPTGB_LAUNCH();
        return IPT_CUDA_SUCCESS;
    }
    ~MlpCorrection() override { ops.release(); }
};

}  // namespace

// Records (features, target, weight) rows while returning the plain
// diagonal correction, so the solver follows the plain trajectory; with
// `params` set it returns the learned correction instead, so that rows are
// recorded along the learned trajectory (for a further round of training).
struct MlpCollector final : LearnedCorrection {
    const float *params = nullptr;
    const double *Xstar = nullptr;
    int kstar = 0;
    const double *sigma = nullptr;
    double hnorm = 1.0;
    float *out = nullptr;
    long long capacity = 0;
    long long count = 0;
    BlockOps ops;
    DeviceBuffer<double> tn, Xs, O, dots, sgn_d, alpha_d, E, G, U, B, Tp, Up;
    DeviceBuffer<int> lidx_d;
    DeviceBuffer<long long> slot_d;
    void bind(const double *row_coupling, double h) override
    {
        sigma = row_coupling;
        hnorm = h;
    }
    bool learned() const override { return false; }
    int correct(const CorrectionArgs &a, double *T) override
    {
        cudaStream_t s = ops.stream;
        const int c = a.nsel;
        const int n = a.n;
        if (count + (long long)a.nsel * a.n > capacity || sigma == nullptr) {
            return ops.diag_correction(a.R, a.d, a.theta, a.sel, a.nsel, a.n, a.clip, T);
        }
        if (tn.count < (size_t)c) {
            IPTGB_CHECK(tn.alloc((size_t)c, s));
            IPTGB_CHECK(dots.alloc(3 * (size_t)c, s));
            IPTGB_CHECK(sgn_d.alloc((size_t)c, s));
            IPTGB_CHECK(alpha_d.alloc((size_t)c, s));
            IPTGB_CHECK(lidx_d.alloc((size_t)c, s));
            IPTGB_CHECK(slot_d.alloc((size_t)c, s));
            IPTGB_CHECK(O.alloc((size_t)kstar * c, s));
        }
        if (Xs.count < (size_t)n * c) {
            IPTGB_CHECK(Xs.alloc((size_t)n * c, s));
            IPTGB_CHECK(E.alloc((size_t)n * c, s));
            IPTGB_CHECK(B.alloc((size_t)n * c, s));
            IPTGB_CHECK(Tp.alloc((size_t)n * c, s));
            IPTGB_CHECK(Up.alloc((size_t)n * c, s));
        }
        IPTGB_CHECK(plain_and_second_order(ops, a, T, U, tn.ptr));
        // overlaps of the current Ritz vectors with the converged ones
        IPTGB_CHECK(ops.gather_columns(a.X, n, a.sel, nullptr, n, c, Xs.ptr, n));
        IPTGB_CHECK(ops.gram(Xstar, n, kstar, Xs.ptr, n, c, n, O.ptr, kstar));
        std::vector<double> hO((size_t)kstar * c);
        IPTGB_CUDA(cudaMemcpyAsync(hO.data(), O.ptr, hO.size() * sizeof(double),
                                   cudaMemcpyDeviceToHost, s));
        IPTGB_CUDA(cudaStreamSynchronize(s));
        std::vector<int> li((size_t)c);
        std::vector<double> sg((size_t)c);
        for (int q = 0; q < c; ++q) {
            int best = 0;
            for (int l = 1; l < kstar; ++l) {
                if (fabs(hO[(size_t)q * kstar + l]) > fabs(hO[(size_t)q * kstar + best])) best = l;
            }
            li[(size_t)q] = best;
            sg[(size_t)q] = hO[(size_t)q * kstar + best] < 0.0 ? -1.0 : 1.0;
        }
        IPTGB_CUDA(cudaMemcpyAsync(lidx_d.ptr, li.data(), (size_t)c * sizeof(int),
                                   cudaMemcpyHostToDevice, s));
        IPTGB_CUDA(cudaMemcpyAsync(sgn_d.ptr, sg.data(), (size_t)c * sizeof(double),
                                   cudaMemcpyHostToDevice, s));
        mlp::collect_error_kernel<<<blocks_for((size_t)n * c), kThreads, 0, s>>>(
            Xstar, lidx_d.ptr, sgn_d.ptr, a.X, a.sel, c, n, E.ptr);
        IPTGB_LAUNCH();
        // keep only the part of the error outside the search space (two
        // passes), and fit it by the projected two-term correction t1 + u
        for (int pass = 0; pass < 2; ++pass) IPTGB_CHECK(project_out(ops, a, E.ptr, G));
        IPTGB_CUDA(cudaMemcpyAsync(B.ptr, T, (size_t)n * c * sizeof(double),
                                   cudaMemcpyDeviceToDevice, s));
        mlp::add_kernel<<<blocks_for((size_t)n * c), kThreads, 0, s>>>(B.ptr, U.ptr,
                                                                      (size_t)n * c);
        IPTGB_LAUNCH();
        IPTGB_CHECK(project_out(ops, a, B.ptr, G));
        // the projected t1 and u of the per-row targets
        IPTGB_CUDA(cudaMemcpyAsync(Tp.ptr, T, (size_t)n * c * sizeof(double),
                                   cudaMemcpyDeviceToDevice, s));
        IPTGB_CUDA(cudaMemcpyAsync(Up.ptr, U.ptr, (size_t)n * c * sizeof(double),
                                   cudaMemcpyDeviceToDevice, s));
        for (int pass = 0; pass < 2; ++pass) {
            IPTGB_CHECK(project_out(ops, a, Tp.ptr, G));
            IPTGB_CHECK(project_out(ops, a, Up.ptr, G));
        }
        mlp::collect_dots_kernel<<<c, 256, 0, s>>>(E.ptr, B.ptr, n, dots.ptr);
        IPTGB_LAUNCH();
        std::vector<double> hd(3 * (size_t)c);
        IPTGB_CUDA(cudaMemcpyAsync(hd.data(), dots.ptr, hd.size() * sizeof(double),
                                   cudaMemcpyDeviceToHost, s));
        IPTGB_CUDA(cudaStreamSynchronize(s));
        std::vector<double> al((size_t)c, 1.0);
        std::vector<long long> slot((size_t)c, -1);
        for (int q = 0; q < c; ++q) {
            const double et = hd[3 * (size_t)q], tt = hd[3 * (size_t)q + 1],
                         ee = hd[3 * (size_t)q + 2];
            // skip pairs whose exact correction is (numerically) orthogonal to
            // the two-term one, or already converged
            if (!(tt > 0.0) || !(ee > 1e-28) || fabs(et) < 0.05 * sqrt(tt * ee)) continue;
            al[(size_t)q] = et / tt;
            slot[(size_t)q] = count;
            count += n;
        }
        IPTGB_CUDA(cudaMemcpyAsync(alpha_d.ptr, al.data(), (size_t)c * sizeof(double),
                                   cudaMemcpyHostToDevice, s));
        IPTGB_CUDA(cudaMemcpyAsync(slot_d.ptr, slot.data(), (size_t)c * sizeof(long long),
                                   cudaMemcpyHostToDevice, s));
        mlp::collect_rows_kernel<<<blocks_for((size_t)n * c), kThreads, 0, s>>>(
            E.ptr, alpha_d.ptr, slot_d.ptr, U.ptr, a.X, a.d, a.theta, a.sel, c, n, a.clip, hnorm,
            sigma, tn.ptr, a.rnorm, T, Tp.ptr, Up.ptr, out);
        IPTGB_LAUNCH();
        if (params != nullptr) {
            mlp::mlp_correct_kernel<<<blocks_for((size_t)n * c), 256, 0, s>>>(
                params, U.ptr, a.X, a.d, a.theta, a.sel, c, n, a.clip, hnorm, sigma, tn.ptr,
                a.rnorm, T);
            IPTGB_LAUNCH();
        }
        IPTGB_CUDA(cudaStreamSynchronize(s));
        return IPT_CUDA_SUCCESS;
    }
    ~MlpCollector() override { ops.release(); }
};

LearnedCorrection *make_learned_correction(const float *params, cudaStream_t stream)
{
    if (params == nullptr) return nullptr;
    auto *m = new MlpCorrection();
    m->params = params;
    m->ops.stream = stream;
    m->ops.sms = device_sm_count();
    return m;
}

LearnedCorrection *make_mlp_collector(const double *Xstar, int kstar, float *out,
                                      long long capacity, const float *params, cudaStream_t stream)
{
    auto *m = new MlpCollector();
    m->params = params;
    m->Xstar = Xstar;
    m->kstar = kstar;
    m->out = out;
    m->capacity = capacity;
    m->ops.stream = stream;
    m->ops.sms = device_sm_count();
    return m;
}

long long mlp_collector_count(const LearnedCorrection *c)
{
    const auto *m = dynamic_cast<const MlpCollector *>(c);
    return m != nullptr ? m->count : 0;
}

}  // namespace iptgb

// ---------------------------------------------------------------------------
// C ABI of the learned preconditioner (include/ipt_block.h)
// ---------------------------------------------------------------------------
using namespace iptgb;

#define IPT_API extern "C" __attribute__((visibility("default")))

IPT_API int ipt_block_mlp_param_count(void) { return mlp::kParams; }

IPT_API int ipt_block_mlp_init(float *d_params, unsigned long long seed, void *stream)
{
    if (d_params == nullptr) return IPT_CUDA_INVALID_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    mlp::mlp_init_kernel<<<blocks_for(mlp::kParams), kThreads, 0, s>>>(d_params, seed);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

IPT_API int ipt_block_mlp_forward(const float *d_params, const float *d_rows, long long rows,
                                  int row_stride, float *d_out, void *stream)
{
    if (d_params == nullptr || d_rows == nullptr || d_out == nullptr || rows < 0 ||
        row_stride < mlp::kIn) {
        return IPT_CUDA_INVALID_ARGUMENT;
    }
    if (rows == 0) return IPT_CUDA_SUCCESS;
    cudaStream_t s = (cudaStream_t)stream;
    mlp::mlp_forward_rows_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, s>>>(
        d_params, d_rows, rows, row_stride, d_out);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

IPT_API int ipt_block_mlp_loss_grad(const float *d_params, const float *d_rows, long long rows,
                                    float *d_grad, void *stream)
{
    if (d_params == nullptr || d_rows == nullptr || d_grad == nullptr || rows <= 0 ||
        rows > (1LL << 30)) {
        return IPT_CUDA_INVALID_ARGUMENT;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int batch = (int)rows;
    const int tiles = mlp::fb_tiles(batch);
    DeviceBuffer<float> part;
    IPTGB_CHECK(part.alloc((size_t)tiles * (mlp::kParams + 1), s));
    IPTGB_CHECK(mlp::launch_fwd_bwd(d_params, d_rows, rows, batch, 0, 0, 0, part.ptr, s));
    mlp::mlp_grad_finish_kernel<<<blocks_for(mlp::kParams + 1, 32), mlp::kSumThreads, 0, s>>>(
        part.ptr, tiles, batch, d_grad);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

IPT_API int ipt_block_mlp_train(float *d_params, const float *d_rows, long long rows, int steps,
                                int batch, float lr, unsigned long long seed,
                                float *d_loss_history, void *stream)
{
    if (d_params == nullptr || d_rows == nullptr || rows <= 0 || steps < 0 || batch <= 0 ||
        batch > (1 << 20) || !(lr > 0.f)) {
        return IPT_CUDA_INVALID_ARGUMENT;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int tiles = mlp::fb_tiles(batch);
    DeviceBuffer<float> part, mv;
    IPTGB_CHECK(part.alloc((size_t)tiles * (mlp::kParams + 1), s));
    IPTGB_CHECK(mv.alloc(2 * (size_t)mlp::kParams, s));
    IPTGB_CUDA(cudaMemsetAsync(mv.ptr, 0, 2 * (size_t)mlp::kParams * sizeof(float), s));
    KernelTimerScope timer(kProfMlp, s);
    for (int it = 1; it <= steps; ++it) {
        IPTGB_CHECK(mlp::launch_fwd_bwd(d_params, d_rows, rows, batch, 1, seed, it, part.ptr, s));
        mlp::mlp_adam_kernel<<<blocks_for(mlp::kParams + 1, 32), mlp::kSumThreads, 0, s>>>(
            d_params, mv.ptr, mv.ptr + mlp::kParams, part.ptr, tiles, batch, it, lr,
            d_loss_history);
        IPTGB_LAUNCH();
    }
    return IPT_CUDA_SUCCESS;
}
