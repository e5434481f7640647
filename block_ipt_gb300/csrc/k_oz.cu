// k_oz.cu - FP64-accurate block product Y = H X on the FP16 tensor cores.
//
// Replaces the reference's FP64 cublasDgemm of the plain IPT loop
// (IPT_C_GPU/src/ipt_cuda.cu:1649,1888), of the mixed refinement
// (IPT_C_GPU/src/mixed_precision/ipt_mixed_precision_cuda.cu:917,958) and of
// the Rayleigh-Ritz products.  H = D + Delta: the diagonal part is applied
// in FP64, Delta X by the split-operand scheme of oz.cuh.
//
// oz_product_kernel<S, CP, MODE> is persistent, one CTA per SM over a
// contiguous range of (column group, 128-row tile, K period) items, in stages
// of 32 K elements, with a warp role for each resource:
//  * warp 18 streams the digit words of Delta (8 bytes per entry, written once
//    per solve) by 32 KB bulk copies; without words (one-off products, very
//    large n) the converters copy the entries of H themselves (cp.async);
//  * warps 0-7, the converters, expand the words into S FP16 digits per entry
//    (one byte permute and one subtraction per two digits; from entries of H
//    ~25 integer instructions more) and store 16-byte runs into the stage's
//    64-byte-swizzled K-major A slices.  The words of the next stage are read
//    before the current one is stored;
//  * warp 16 brings the S x CP digit rows of X by TMA;
//  * warp 17 issues tcgen05.mma: per slice s and 16-element K step one MMA of
//    N = (slices t with s + t < V) * CP that adds every pair (s, t) into the
//    TMEM accumulator of level s + t (the B slices are consecutive rows, the
//    level accumulators consecutive columns): few and wide MMAs, since each
//    costs its issuing thread tens of cycles;
//  * warps 8-15 drain the level accumulators after every period (two sets, so
//    the next period's MMAs run meanwhile, when they fit in TMEM).  S = 7 adds
//    the levels as 96-bit integers, moved to the largest of the scales that
//    the row's and the column's blocks of 128 entries have; S = 6 combines
//    them in double-float arithmetic.  A CTA leaving a tile writes one FP64
//    partial.
// The consumer of the partials (oz_finish_kernel or oz_update_kernel) adds
// those of a tile in a fixed order, so the product is deterministic.
//
// What bounds it: shared-memory bandwidth.  A stage moves 32 KB of words in
// and out, 56 KB (S = 7) of digits in and, through the MMAs, out again, and
// the MMAs read the digit rows of X 34 times 2 KB: 265 KB, 2070 cycles at 128
// bytes per cycle, against 1090 cycles of MMA and 32 KB of HBM traffic (79 us
// per product of n = 8192 at the measured 6.8 TB/s).  Measured at n = 8192, 32
// columns: 132 us per product with one scale per row and column (2240 cycles
// per stage; tensor pipe 50 %, HBM 54 %), 147 us with those of S = 7 (35 more
// instructions per sum in the drain); the split-K FP64 SIMT product it replaces
// in the plain path 3.6 ms (95 % of the FP64 pipe).  With one scale: digit
// slices stored as FP16 (14 bytes per entry with 7 slices) would need 139 us of
// HBM time; extracting the digits from H in every product took 205 us (55
// instructions per entry); A operands in TMEM instead of shared memory 137 us
// (their tcgen05.st wait for the MMAs, and only one accumulator set fits).
//
// Every mbarrier wait is bounded; a timeout sets the error flag, the CTA
// drains its own copies and MMAs (bounded), frees TMEM and returns.
#include <cuda.h>
#include <cuda_fp16.h>
#include <float.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <climits>

#include "common.cuh"
#include "ipt_plain.h"
#include "kernels.cuh"
#include "oz.cuh"
#include "oz_product.h"
#include "reduce.cuh"
#include "tcgen05.cuh"
#include "thread_slots.h"

namespace iptgb {

namespace oz {

constexpr int kBM = 128;                       // UMMA M: rows per tile
constexpr int kStageK = 32;                    // K elements per stage (64 B of FP16)
constexpr uint32_t kABytes = kBM * 64;         // one slice of one stage: 8 KB
constexpr int kConvWarps = 8;                  // warps 0-7: digits into the A ring
constexpr int kDrainWarps = 8;                 // warps 8-15: accumulators to running sums
constexpr int kProducerWarp = kConvWarps + kDrainWarps;
constexpr int kMmaWarp = kProducerWarp + 1;
constexpr int kWordsWarp = kProducerWarp + 2;
constexpr int kThreads = 32 * (kConvWarps + kDrainWarps + 3);
constexpr int kStages = 2;                     // A ring depth
constexpr int kMaxBStages = 3;                 // B ring depth, where shared memory allows
constexpr int kRawStages = 2;                  // ring of digit words / H entries
constexpr uint32_t kRawBytes = kBM * kStageK * 8;
constexpr int kMaxStagesPerItem = kOzPeriod / kStageK;
// a matrix below this size stays in L2 between the products of a solve (126
// MB usable); larger ones are streamed past it
constexpr size_t kL2ResidentBytes = 96u << 20;

// Where the digits come from: kWords - digit words written once per solve
// (OzMatrix::words), 32 KB blocks by bulk copies; kRows - the entries of H
// themselves, by each converter thread's own cp.async copies (one-off
// products, and matrices whose digit words would take too much memory).
enum Mode { kRows = 0, kWords = 1 };

struct Params {
    const double *H;
    const uint4 *words;
    const int *rowexp;    // S = 6: per row
    // S = 7: biased exponents (oz_pack_exponent) of Delta, [block][row], and of
    // X, [group][block][CP], two to a word
    const uint16_t *blockexp;
    const uint32_t *xexp;
    int blocks;           // of kOzBlock K elements
    int n, groups, tiles, periods, nstages;  // nstages: K stages of a row
    int spp;         // stages per period (item): at most kMaxStagesPerItem
    long long items;
    int maxslots;
    int stream_h;    // H is read past L2 (evict first)
    int b_loads;     // TMA boxes per B stage
    uint32_t b_bytes;
    long long spin;  // polls of a pipeline wait before it gives up
};

template <int S, int CP>
struct Layout {
    static constexpr int V = OzSplit<S>::kLevels;
    static constexpr int kSets = 2 * V * CP <= 512 ? 2 : 1;  // accumulator sets in TMEM
    static constexpr uint32_t kA = S * kABytes;    // A digits of a stage
    static constexpr uint32_t kB = S * CP * 64;    // B digits of a stage
    static constexpr uint32_t kFixed = 1024 + kStages * kA + kRawStages * kRawBytes;
    static constexpr int kBStages = kFixed + kMaxBStages * kB + 512 <= 227 * 1024 ? kMaxBStages : 2;
    static constexpr uint32_t kSmem = kFixed + kBStages * kB;
    static_assert(kSmem + 512 <= 227 * 1024, "shared memory");
};

using tc::owner_of;

__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// Instruction descriptor without N: M = 128, FP16 x FP16 -> FP32.
constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(kBM >> 4) << 24);

// K-major operand, 64-byte swizzle: rows of 64 bytes, 8-row atoms of 512
// bytes, descriptor version 1.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)(16u >> 4) << 16;
    d |= (uint64_t)(512u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

// Asynchronous copies of H entries into a converter thread's own slots
// (`bytes` 0 writes zeros).
__device__ __forceinline__ void copy8(uint32_t dst, const double *src, int bytes, uint64_t pol)
{
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 8, %2, %3;" ::"r"(dst),
                 "l"(src), "r"(bytes), "l"(pol)
                 : "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes,
                                          uint32_t bar, uint64_t pol)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1], %2, [%3], %4;" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar), "l"(pol)
        : "memory");
}

__device__ __forceinline__ uint64_t l2_normal_policy()
{
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

// Position in a CTA's sequence of stages: item it = (group * tiles + tile) *
// periods + per, stage st of its period.
struct Walk {
    long long it;
    int grp, tile, per, st, count;  // count: stages of this period
    __device__ __forceinline__ void start(long long first, const Params &p)
    {
        it = first;
        per = (int)(first % p.periods);
        tile = (int)((first / p.periods) % p.tiles);
        grp = (int)(first / ((long long)p.periods * p.tiles));
        st = 0;
        count = min(p.spp, p.nstages - per * p.spp);
    }
    __device__ __forceinline__ void next(const Params &p)
    {
        if (++st < count) return;
        st = 0;
        ++it;
        if (++per == p.periods) {
            per = 0;
            if (++tile == p.tiles) {
                tile = 0;
                ++grp;
            }
        }
        count = min(p.spp, p.nstages - per * p.spp);
    }
    // to the next item
    __device__ __forceinline__ void skip(const Params &p)
    {
        st = count - 1;
        next(p);
    }
};

// Starts the copies of a thread's eight K entries l0..l0+7 of row `row` of H
// (zeros outside the matrix) into its slots of the raw tile [32 K][128 rows].
__device__ __forceinline__ void fetch8(const Params &p, const Walk &w, int r, int g, uint64_t pol,
                                       uint32_t raw)
{
    const int row0 = w.tile * kBM;
    const int row = row0 + r;
    const int k0 = (w.per * p.spp + w.st) * kStageK;
    const int l0 = k0 + 8 * g;
    if (row0 + kBM <= p.n && k0 + kStageK <= p.n) {
        const double *h = p.H + (size_t)l0 * p.n + row;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            copy8(raw + (uint32_t)(u * kBM * 8), h, 8, pol);
            h += p.n;
        }
    } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int l = l0 + u;
            const bool in = row < p.n && l < p.n;
            copy8(raw + (uint32_t)(u * kBM * 8), in ? p.H + (size_t)l * p.n + row : p.H,
                  in ? 8 : 0, pol);
        }
    }
}

__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}

// Waits for the TMEM loads issued so far; naming the registers they fill keeps
// every use of them behind the wait.
template <int V, int N>
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[V][N])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int l = 0; l < V; ++l) {
#pragma unroll
        for (int j = 0; j < N; ++j) asm volatile("" : "+r"(r[l][j])::"memory");
    }
}

// v 2^e; one multiplication where 2^e is a normal number.
__device__ __forceinline__ double scale2(double v, int e)
{
    if (e > -1022 && e < 1023) return v * __hiloint2double((e + 1023) << 20, 0);
    return ldexp(v, e);
}

// Running sums of a thread's columns over the periods of a tile.
template <int S, int NC>
struct Sums;
// 56-bit split: 96-bit integers (three words; a pair of 64-bit sums would not
// leave the drain's loads enough registers) in units of 2^(E + kOut), E at
// least the exponent of every product so far.  Per period the levels 0-3 and
// 4-7 are each combined by one wide multiply-add per level into 64 bits (below
// 2^48), with weights 2^24, 2^16, 2^8, 1; the sum, below 2^80, moves down to
// the unit.  Exponents are pairs of biased 16-bit ones (two columns;
// oz_pack_exponent), so that one addition or subtraction serves both.
template <int NC>
struct Sums<7, NC> {
    uint32_t w[NC][3];
    uint32_t E[NC / 2];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int j = 0; j < NC; ++j) w[j][0] = w[j][1] = w[j][2] = 0;
#pragma unroll
        for (int j = 0; j < NC / 2; ++j) E[j] = 0;
    }
    // columns 4, 5, ... become columns 0, 1, ...
    __device__ __forceinline__ void rotate()
    {
        uint32_t t[4][3];
        const uint32_t e0 = E[0], e1 = E[1];
#pragma unroll
        for (int j = 0; j < NC; ++j) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if (j < 4) t[j][q] = w[j][q];
                w[j][q] = j + 4 < NC ? w[j + 4 < NC ? j + 4 : j][q] : t[j + 4 - NC][q];
            }
        }
#pragma unroll
        for (int j = 0; j + 2 < NC / 2; ++j) E[j] = E[j + 2];
        E[NC / 2 - 2] = e0;
        E[NC / 2 - 1] = e1;
    }
    // x down by `bits` (at most 95)
    static __device__ __forceinline__ void shift(uint32_t (&x)[3], uint32_t bits)
    {
        const uint32_t sign = (uint32_t)((int)x[2] >> 31);
        const bool two = bits >= 64, one = (bits & 32) != 0;
        const uint32_t u0 = two ? x[2] : x[0], u1 = two ? sign : x[1], u2 = two ? sign : x[2];
        const uint32_t v0 = one ? u1 : u0, v1 = one ? u2 : u1, v2 = one ? sign : u2;
        x[0] = __funnelshift_r(v0, v1, bits);
        x[1] = __funnelshift_r(v1, v2, bits);
        x[2] = (uint32_t)((int)v2 >> (bits & 31));
    }
    // Units for products of exponents e(j) (pairs).  One that has to rise goes
    // kSpare binades beyond: the next rise is seldom then (entries that grow
    // towards the diagonal), and 2^-66 is far below the operands' 2^-56.
    static constexpr uint32_t kSpare = 6u | 6u << 16;
    template <typename F>
    __device__ __forceinline__ void raise(F e)
    {
        uint32_t above = 0;  // (e() is warp-collective)
#pragma unroll
        for (int j = 0; j < NC / 2; ++j) above |= __vmaxu2(E[j], e(j)) ^ E[j];
        if (!__any_sync(0xffffffffu, above != 0)) return;
#pragma unroll
        for (int j = 0; j < NC / 2; ++j) {
            // (0 or the new unit, per half)
            const uint32_t ej = e(j);
            const uint32_t up = __vcmpgtu2(ej, E[j]);
            const uint32_t now = ((ej + kSpare) & up) | (E[j] & ~up);
            const uint32_t by = __vminu2(now - E[j], 95u | 95u << 16);
            E[j] = now;
            shift(w[2 * j], by & 0xFFFFu);
            shift(w[2 * j + 1], by >> 16);
        }
    }
    // v + x w, on the multiply pipe (the integer one is the converters')
    static __device__ __forceinline__ long long mad(int x, int w, long long v)
    {
        asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(v) : "r"(x), "r"(w));
        return v;
    }
    static __device__ __forceinline__ long long combine(uint32_t l0, uint32_t l1, uint32_t l2,
                                                        uint32_t l3)
    {
        long long v = mad(__float2int_rn(__uint_as_float(l3)), 1, 0);
        v = mad(__float2int_rn(__uint_as_float(l2)), 1 << 8, v);
        v = mad(__float2int_rn(__uint_as_float(l1)), 1 << 16, v);
        return mad(__float2int_rn(__uint_as_float(l0)), 1 << 24, v);
    }
    // column j: hi 2^32 + lo, `down` bits (at most 95) below the unit
    __device__ __forceinline__ void add(int j, long long hi, long long lo, uint32_t down)
    {
        const long long top = mad((int)(lo >> 32), 1, hi);
        uint32_t x[3] = {(uint32_t)lo, (uint32_t)top, (uint32_t)(top >> 32)};
        shift(x, down);
        asm("add.cc.u32 %0, %0, %3;\n\t"
            "addc.cc.u32 %1, %1, %4;\n\t"
            "addc.u32 %2, %2, %5;"
            : "+r"(w[j][0]), "+r"(w[j][1]), "+r"(w[j][2])
            : "r"(x[0]), "r"(x[1]), "r"(x[2]));
    }
    __device__ __forceinline__ double value(int j) const
    {
        const long long hi = (long long)(((uint64_t)w[j][2] << 32) | w[j][1]);
        const int e = (int)((j & 1) != 0 ? E[j >> 1] >> 16 : E[j >> 1] & 0xFFFFu);
        return scale2((double)hi * 4294967296.0 + (double)w[j][0],
                      e + 2 * kOzZeroExp + OzSplit<7>::kOut);
    }
};
// 48-bit split: double-float (H, L).
template <int NC>
struct Sums<6, NC> {
    float H[NC], L[NC];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int j = 0; j < NC; ++j) H[j] = L[j] = 0.0f;
    }
    __device__ __forceinline__ void add(int j, const uint32_t (&l)[6])
    {
        float v[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = __uint_as_float(l[q]);
        float h, hh, e1, e2;
        two_sum(v[0], v[1] * 0x1p-8f, h, e1);
        two_sum(h, v[2] * 0x1p-16f, hh, e2);
        const float ll = e1 + e2;
        const float t = ll + (v[3] * 0x1p-24f + (v[4] * 0x1p-32f + v[5] * 0x1p-40f));
        float s, e;
        two_sum(H[j], hh, s, e);
        H[j] = s;
        L[j] += t + e;
    }
    __device__ __forceinline__ double value(int j) const { return (double)H[j] + (double)L[j]; }
};

template <int S, int CP, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
oz_product_kernel(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ Params prm,
                  double *__restrict__ P, int *err)
{
    using Lay = Layout<S, CP>;
    constexpr int V = Lay::V;
    constexpr int kSets = Lay::kSets;
    constexpr int NC = CP / 2;                        // columns a drain warp sums
    constexpr uint32_t kBBytes = Lay::kB;
    constexpr int kBStages = Lay::kBStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
    __shared__ uint64_t bars[2 * kStages + 2 * kBStages + 2 * kRawStages + 5];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ int b_issued, h_issued;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const long long G = gridDim.x;
    const long long it0 = (long long)blockIdx.x * prm.items / G;
    const long long it1 = ((long long)blockIdx.x + 1) * prm.items / G;
    const uint32_t bar0 = tc::smem_u32(bars);
    auto bar = [&](int q) { return bar0 + 8u * (uint32_t)q; };
    auto a_full = [&](int q) { return bar(q); };
    auto a_empty = [&](int q) { return bar(kStages + q); };
    auto b_full = [&](int q) { return bar(2 * kStages + q); };
    auto b_empty = [&](int q) { return bar(2 * kStages + kBStages + q); };
    constexpr int kRawBar = 2 * kStages + 2 * kBStages;
    auto raw_full = [&](int q) { return bar(kRawBar + q); };
    auto raw_empty = [&](int q) { return bar(kRawBar + kRawStages + q); };
    constexpr int kAccBar = kRawBar + 2 * kRawStages;
    auto acc_full = [&](int b) { return bar(kAccBar + b); };
    auto acc_empty = [&](int b) { return bar(kAccBar + 2 + b); };
    const uint32_t mma_done = bar(kAccBar + 4);
    const uint32_t base = tc::smem_u32(smem);
    const uint32_t b0 = base + kStages * Lay::kA;
    const uint32_t raw0 = b0 + kBStages * kBBytes;

    if (threadIdx.x == 0) {
        for (int q = 0; q < kStages; ++q) {
            tc::mbar_init(a_full(q), kConvWarps);
            tc::mbar_init(a_empty(q), 1);
        }
        for (int q = 0; q < kBStages; ++q) {
            tc::mbar_init(b_full(q), 1);
            tc::mbar_init(b_empty(q), 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(acc_full(b), 1);
            tc::mbar_init(acc_empty(b), kDrainWarps);
        }
        for (int q = 0; q < kRawStages; ++q) {
            tc::mbar_init(raw_full(q), 1);
            tc::mbar_init(raw_empty(q), kConvWarps);
        }
        tc::mbar_init(mma_done, 1);
        abort_flag = 0;
        b_issued = 0;
        h_issued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kProducerWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         tc::smem_u32(&tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp == kProducerWarp) {
        if (lane == 0) {
            // ---- TMA producer: the digit rows of X, one stage at a time ----
            pdl_wait();  // the grid that wrote them
            int q = 0, issued = 0;
            uint32_t par = 0;
            Walk w;
            w.start(it0, prm);
            while (w.it < it1 && !abort_flag) {
                if (issued >= kBStages && !tc::mbar_wait(b_empty(q), par ^ 1u, err, 12, false, prm.spin)) {
                    abort_flag = 1;
                    break;
                }
                const uint32_t dst = b0 + (uint32_t)q * kBBytes;
                const int x = (w.per * prm.spp + w.st) * kStageK;
                const int y = w.grp * S * CP;
                tc::mbar_expect_tx(b_full(q), prm.b_bytes);
                tc::tma_load_2d(dst, &tmB, x, y, b_full(q));
                if (prm.b_loads == 2) {
                    tc::tma_load_2d(dst + (uint32_t)(S / 2 * CP * 64), &tmB, x, y + S / 2 * CP,
                                    b_full(q));
                }
                ++issued;
                if (++q == kBStages) {
                    q = 0;
                    par ^= 1u;
                }
                w.next(prm);
            }
            b_issued = issued;
        }
    } else if (warp == kWordsWarp) {
        if (MODE == kWords && lane == 0) {
            // ---- producer of the digit words (which no preceding kernel of
            // the iteration writes), as far ahead as the converters free the
            // ring ----
            const uint64_t pol = prm.stream_h ? tc::l2_stream_policy() : l2_normal_policy();
            int q = 0, issued = 0;
            uint32_t par = 0;
            Walk w;
            w.start(it0, prm);
            while (w.it < it1 && !abort_flag) {
                if (issued >= kRawStages &&
                    !tc::mbar_wait(raw_empty(q), par ^ 1u, err, 10, false, prm.spin)) {
                    abort_flag = 1;
                    break;
                }
                const size_t block = (size_t)w.tile * prm.nstages + (w.per * prm.spp + w.st);
                tc::mbar_expect_tx(raw_full(q), kRawBytes);
                bulk_load(raw0 + (uint32_t)q * kRawBytes, prm.words + block * (kRawBytes / 16),
                          kRawBytes, raw_full(q), pol);
                ++issued;
                if (++q == kRawStages) {
                    q = 0;
                    par ^= 1u;
                }
                w.next(prm);
            }
            h_issued = issued;
        }
    } else if (warp == kMmaWarp) {
        // ---- tcgen05.mma issuer: the whole warp walks the stages, one
        // elected lane issues (see umma_f16_elect) ----
        int q = 0, bq = 0;
        uint32_t par = 0, bpar = 0;
        bool ok = true;
        Walk w;
        w.start(it0, prm);
        for (int k = 0; ok && w.it < it1; ++k) {
            // accumulator set k % kSets: wait until its previous use (item
            // k - kSets) has been drained
            const int ab = k % kSets;
            const int use = k / kSets;
            if (use > 0) {
                ok = __all_sync(0xffffffffu, tc::mbar_wait(acc_empty(ab), (uint32_t)((use - 1) & 1),
                                                           err, 13, false, prm.spin));
                if (!ok) break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + (uint32_t)(ab * V * CP);
            const long long item = w.it;
            bool first = true;
            while (w.it == item) {
                ok = tc::mbar_wait(b_full(bq), bpar, err, 14, false, prm.spin) &&
                     tc::mbar_wait(a_full(q), par, err, 15, false, prm.spin);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t ad0 = sw64_desc(base + (uint32_t)q * Lay::kA);
                const uint64_t bd0 = sw64_desc(b0 + (uint32_t)bq * kBBytes);
#pragma unroll
                for (int kk = 0; kk < kStageK / 16; ++kk) {
                    // the first K step of an item initialises the
                    // accumulators: slice 0 those of its S levels, and
                    // (V > S) slice 1 the one of level S
                    const uint32_t acc_on = first && kk == 0 ? 0u : 1u;
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        constexpr uint32_t kColStep = (uint32_t)(CP * 64) >> 4;
                        const int nt = S < V - s ? S : V - s;
                        const uint64_t ad =
                            ad0 + (uint64_t)(s * (int)(kABytes >> 4) + 2 * kk);
                        const uint64_t bd = bd0 + (uint64_t)(2 * kk);
                        const uint32_t dst = acc + (uint32_t)(s * CP);
                        auto mma = [&](int t0, int count, uint32_t accum) {
                            tc::umma_f16_elect(dst + (uint32_t)(t0 * CP), ad,
                                               bd + (uint64_t)(t0 * kColStep),
                                               kIdesc | ((uint32_t)(count * CP) >> 3 << 17),
                                               accum);
                        };
                        if (V > S && s == 1) {
                            // level S starts here: its pair (1, S - 1) apart
                            if (acc_on == 0u) {
                                mma(0, nt - 1, 1u);
                                mma(nt - 1, 1, 0u);
                            } else {
                                mma(0, nt, 1u);
                            }
                        } else if (nt * CP > 256) {
                            mma(0, nt / 2, s == 0 ? acc_on : 1u);
                            mma(nt / 2, nt - nt / 2, s == 0 ? acc_on : 1u);
                        } else {
                            mma(0, nt, s == 0 ? acc_on : 1u);
                        }
                    }
                }
                tc::umma_commit_elect(a_empty(q));
                tc::umma_commit_elect(b_empty(bq));
                if (++q == kStages) {
                    q = 0;
                    par ^= 1u;
                }
                if (++bq == kBStages) {
                    bq = 0;
                    bpar ^= 1u;
                }
                first = false;
                w.next(prm);
            }
            if (ok) tc::umma_commit_elect(acc_full(ab));
        }
        if (!ok) abort_flag = 1;
        tc::umma_commit_elect(mma_done);
    } else if (warp < kConvWarps) {
        // ---- converters: a thread converts two runs of 8 K entries (groups
        // g0 and g0 + 1 of the stage's four) of row r, lanes = rows ----
        const int r = (int)threadIdx.x & 127;
        const int g0 = 2 * ((int)threadIdx.x >> 7);
        const uint64_t pol = prm.stream_h ? tc::l2_stream_policy() : l2_normal_policy();
        const uint32_t my_raw = (uint32_t)(8 * g0 * kBM + r) * 8u;  // kRows
        Walk w, lw;  // conversion and copy positions
        w.start(it0, prm);
        lw = w;
        auto fetch = [&](int q) {  // kRows: the copies of the next stage, one group
            if (lw.it < it1) {
                fetch8(prm, lw, r, g0, pol, raw0 + (uint32_t)q * kRawBytes + my_raw);
                fetch8(prm, lw, r, g0 + 1, pol,
                       raw0 + (uint32_t)q * kRawBytes + my_raw + 8u * kBM * 8u);
                lw.next(prm);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (MODE == kRows) {
            for (int q = 0; q < kRawStages; ++q) fetch(q);
        }
        int q = 0, rq = 0, done = 0;
        uint32_t par = 0, rpar = 0;
        int e_row = 0, e_tile = -1, e_block = -1;
        bool good = true;
        // the packed digits of this thread's 16 K entries of the stage at w,
        // which then moves on
        auto load = [&](uint4 (&x)[8]) {
            if (MODE == kWords) {
                if (!__all_sync(0xffffffffu, tc::mbar_wait(raw_full(rq), rpar, err, 9, false, prm.spin))) {
                    good = false;
                    return;
                }
                const uint32_t src = raw0 + (uint32_t)rq * kRawBytes + (uint32_t)(r * 256);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(x[j].x), "=r"(x[j].y), "=r"(x[j].z), "=r"(x[j].w)
                                 : "r"(src + (uint32_t)(((4 * g0 + j) ^ (r & 7)) << 4))
                                 : "memory");
                }
                // the slot may be refilled once every lane's words have arrived:
                // the arrival alone does not wait for loads under way (with more
                // work in the drain warps rows came out wrong, and otherwise in
                // the next run)
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(raw_empty(rq));
            } else {
                const int k0 = (w.per * prm.spp + w.st) * kStageK;
                const int block = S == 7 ? k0 / kOzBlock : 0;
                if (w.tile != e_tile || block != e_block) {
                    e_tile = w.tile;
                    e_block = block;
                    const int row = w.tile * kBM + r;
                    e_row = kOzNonFinite;
                    if (row < prm.n) {
                        e_row = S == 7 ? oz_unpack_exponent(
                                             __ldg(prm.blockexp + (size_t)block * prm.n + row))
                                       : __ldg(prm.rowexp + row);
                    }
                }
                const bool on_diag = k0 < w.tile * kBM + kBM && k0 + kStageK > w.tile * kBM;
                asm volatile("cp.async.wait_group %0;" ::"n"(kRawStages - 1) : "memory");
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    double v[8];
                    const uint32_t src =
                        raw0 + (uint32_t)rq * kRawBytes + my_raw + (uint32_t)(c * 8 * kBM * 8);
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        asm volatile("ld.shared.f64 %0, [%1];"
                                     : "=d"(v[u])
                                     : "r"(src + (uint32_t)(u * kBM * 8))
                                     : "memory");
                    }
                    if (on_diag) {  // Delta leaves the diagonal out
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            if (k0 + 8 * (g0 + c) + u == w.tile * kBM + r) v[u] = 0.0;
                        }
                    }
                    if (e_row >= kOzFastExp) {
                        const int nb = oz_shift_base<S>(e_row);
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            x[4 * c + p] = oz_pack_pair<S>(oz_biased<S>(v[2 * p], nb),
                                                           oz_biased<S>(v[2 * p + 1], nb));
                        }
                    } else {
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            x[4 * c + p] = oz_pack_pair<S>(oz_biased_any<S>(v[2 * p], e_row),
                                                           oz_biased_any<S>(v[2 * p + 1], e_row));
                        }
                    }
                }
                fetch(rq);
            }
            if (++rq == kRawStages) {
                rq = 0;
                rpar ^= 1u;
            }
            w.next(prm);
        };
        // their FP16 digits into the next slot of the A ring, one 16-byte run
        // of K per slice and K group
        auto emit = [&](const uint4 (&x)[8]) {
            if (done >= kStages &&
                !__all_sync(0xffffffffu, tc::mbar_wait(a_empty(q), par ^ 1u, err, 11, false, prm.spin))) {
                good = false;
                return;
            }
            const uint32_t row = base + (uint32_t)q * Lay::kA + (uint32_t)(r * 64);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t dst = row + (uint32_t)(((g0 + c) ^ ((r >> 1) & 3)) << 4);
#pragma unroll
                for (int s = S - 1; s >= 0; --s) {
                    uint32_t h[4];
#pragma unroll
                    for (int p = 0; p < 4; ++p) h[p] = oz_slice_pair<S>(x[4 * c + p], s);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst +
                                                                                  s * kABytes),
                                 "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3])
                                 : "memory");
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(a_full(q));
            ++done;
            if (++q == kStages) {
                q = 0;
                par ^= 1u;
            }
        };
        // the words of the next stage are read before those of the current
        // one are stored
        uint4 xa[8], xb[8];
        if (w.it < it1) load(xa);
        while (good) {
            const bool more = w.it < it1;
            if (more) load(xb);
            if (good) emit(xa);
            if (!more || !good) break;
            const bool again = w.it < it1;
            if (again) load(xa);
            if (good) emit(xb);
            if (!again) break;
        }
        if (!good) abort_flag = 1;
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ---- drain: the level accumulators of every item into running sums,
        // warp = 32 rows x NC columns, and a tile's sums to its partial ----
        const int drow = (warp & 3) * 32 + lane;
        const int dcol = ((warp - kConvWarps) >> 2) * NC;
        Sums<S, NC> sums;
        sums.clear();
        if (S == 7) pdl_wait();  // the exponents of X
        int k = 0;
        Walk w;
        w.start(it0, prm);
        // S = 7: the exponents of the next item's operands (biased: two columns'
        // per word, one word per lane), read one item ahead
        uint32_t er_next = 0, ex_next = 0;
        auto exponents = [&]() {
            if (w.it >= it1) return;
            const int block = w.per * prm.spp / (kOzBlock / kStageK);
            const int row = min(w.tile * kBM + drow, prm.n - 1);
            er_next = (uint32_t)__ldg(prm.blockexp + (size_t)block * prm.n + row);
            ex_next = __ldcg(prm.xexp + (((size_t)w.grp * prm.blocks + block) * CP + dcol) / 2 +
                             lane % (NC / 2));
            w.skip(prm);
        };
        if (S == 7) exponents();
        for (long long it = it0; it < it1; ++it, ++k) {
            const int ab = k % kSets;
            const uint32_t er = er_next | er_next << 16, ex = ex_next;
            if constexpr (S == 7) {
                exponents();
                sums.raise([&](int j) { return er + __shfl_sync(0xffffffffu, ex, j); });
            }
            // warp-uniform decision: the TMEM loads below are warp-collective
            if (!__all_sync(0xffffffffu, tc::mbar_wait(acc_full(ab), (uint32_t)((k / kSets) & 1),
                                                       err, 16, false, prm.spin))) {
                abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t addr =
                tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(ab * V * CP + dcol);
            auto drained = [&]() {
                // the last columns are in registers: the MMAs of a later item
                // may overwrite the set
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(acc_empty(ab));
            };
            if constexpr (S == 7) {
                // four columns and half their levels at a time (more do not fit
                // in the registers): the first four, which then change places
                // with the rest.  (Unrolled, the drain's instructions crowd the
                // converters' out of the instruction cache: 13 us more at n =
                // 8192, 32 columns.)
#pragma unroll 1
                for (int j0 = 0; j0 < NC; j0 += 4) {
                    uint32_t v[4][4];
                    long long hi[4];
                    __syncwarp();  // the loads and their wait are warp-collective
#pragma unroll
                    for (int l = 0; l < 4; ++l) tmem_ld_cols(addr + (uint32_t)(l * CP + j0), v[l]);
                    uint32_t down[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t e = er + __shfl_sync(0xffffffffu, ex, j0 / 2 + j);
                        down[j] = __vminu2(sums.E[j] - e, 95u | 95u << 16);
                    }
                    tmem_ld_wait(v);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        hi[j] = sums.combine(v[0][j], v[1][j], v[2][j], v[3][j]);
                    }
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        tmem_ld_cols(addr + (uint32_t)((4 + l) * CP + j0), v[l]);
                    }
                    tmem_ld_wait(v);
                    if (j0 + 4 >= NC) drained();
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const long long lo = sums.combine(v[0][j], v[1][j], v[2][j], v[3][j]);
                        sums.add(j, hi[j], lo,
                                 (j & 1) != 0 ? down[j >> 1] >> 16 : down[j >> 1] & 0xFFFFu);
                    }
                    sums.rotate();
                }
            } else {
#pragma unroll
                for (int j0 = 0; j0 < NC; j0 += 4) {
                    uint32_t v[V][4];
#pragma unroll
                    for (int l = 0; l < V; ++l) tmem_ld_cols(addr + (uint32_t)(l * CP + j0), v[l]);
                    tmem_ld_wait(v);
                    if (j0 + 4 >= NC) drained();
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t lv[V];
#pragma unroll
                        for (int l = 0; l < V; ++l) lv[l] = v[l][j];
                        sums.add(j0 + j, lv);
                    }
                }
            }
            const long long gt = it / prm.periods;
            if (it + 1 == it1 || (it + 1) / prm.periods != gt) {
                const long long slot =
                    (long long)blockIdx.x - owner_of(gt * prm.periods, prm.items, G);
                double *dst = P + ((size_t)(gt * prm.maxslots + slot) * CP + dcol) * kBM + drow;
#pragma unroll
                for (int j = 0; j < NC; ++j) dst[(size_t)j * kBM] = sums.value(j);
                sums.clear();
            }
        }
    }
    __syncwarp();
    pdl_trigger();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kProducerWarp && lane == 0) {
        // every MMA this CTA issued has completed before TMEM is released
        tc::mbar_wait(mma_done, 0u, err, 17, true);
        if (abort_flag) {
            // drain the copies still in flight (bounded)
            const int bi = b_issued, hi = h_issued;
            for (int i = max(0, bi - kBStages); i < bi; ++i) {
                tc::mbar_wait(b_full(i % kBStages), (uint32_t)((i / kBStages) & 1), err, 18, true);
            }
            for (int i = max(0, hi - kRawStages); i < hi; ++i) {
                tc::mbar_wait(raw_full(i % kRawStages), (uint32_t)((i / kRawStages) & 1), err, 19,
                              true);
            }
        }
    }
    __syncthreads();
    if (warp == kProducerWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                     : "memory");
    }
}

__device__ __forceinline__ unsigned long long abs_bits(double v)
{
    return (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFULL;
}

__device__ __forceinline__ unsigned long long warp_max(unsigned long long m)
{
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, m, off);
        m = o > m ? o : m;
    }
    return m;
}

// Column maxima of |X| as bit patterns (colmax zeroed by the caller): grid
// (column, row chunk), atomicMax per warp.
__global__ void oz_colmax_kernel(const double *__restrict__ X, long long ldx, int n,
                                 unsigned long long *__restrict__ colmax)
{
    pdl_wait();
    const int c = blockIdx.x;
    const double *xc = X + (size_t)c * ldx;
    unsigned long long m = 0;
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < n; j += gridDim.y * blockDim.x) {
        const unsigned long long a = abs_bits(xc[j]);
        m = a > m ? a : m;
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0 && m != 0) atomicMax(colmax + c, m);
    pdl_trigger();
}

// B slices of X: column c = group * cp + j of the padded block holds digit t
// along K in row (group * S + t) * cp + j of B, zero beyond n and for
// c >= C.  Grid (padded column, K chunk); colexp[c] records the column's
// exponent; colmax_next (may be null) is cleared for the pass that writes
// the next block.  S = 7: a warp takes a block of 128 entries, whose exponent
// it leaves in xexp ([group][block][cp]).
//
// With norms.count > 0 an extra block (x = the number of padded columns)
// finishes the norms of the update before, whose blocks only left their parts:
// finished there, by the block with the last ticket, they held up the next
// step by 3 us.
struct PendingNorms {
    const double2 *parts;
    int count;
    double *out;
};

__device__ __forceinline__ void finish_norms(const PendingNorms &p)
{
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < p.count; i += blockDim.x) {
        const double2 v = p.parts[i];
        a += v.x;
        b += v.y;
    }
    write_norms2(block_sum2(a, b), p.out);
}

// The same where no next step follows.
__global__ void __launch_bounds__(256) oz_norms_kernel(PendingNorms norms)
{
    pdl_wait();
    pdl_trigger();
    finish_norms(norms);
}

template <int S>
__global__ void __launch_bounds__(256)
oz_slice_x_kernel(const double *__restrict__ X, long long ldx, int n, int C, int cp, int ldp,
                  const unsigned long long *__restrict__ colmax,
                  unsigned long long *__restrict__ colmax_next, __half *__restrict__ B,
                  int *__restrict__ colexp, uint16_t *__restrict__ xexp, int blocks,
                  PendingNorms norms)
{
    pdl_wait();
    const int c = blockIdx.x;
    if (norms.count > 0 && c == (int)gridDim.x - 1) {
        if (blockIdx.y == 0) finish_norms(norms);
        return;
    }
    const int e = c < C ? oz_exponent(colmax[c]) : 0;
    if (blockIdx.y == 0 && threadIdx.x == 0 && c < C) {
        colexp[c] = e;
        if (colmax_next != nullptr) colmax_next[c] = 0;
    }
    const double *xc = X + (size_t)c * ldx;
    uint2 *row = reinterpret_cast<uint2 *>(B + ((size_t)(c / cp) * S * cp + c % cp) * ldp);
    const size_t stride = (size_t)cp * (size_t)ldp / 4;
    const int lane = threadIdx.x & 31;
    static_assert(kOzBlock == 4 * 32, "one block per warp");
    for (int j0 = 4 * (blockIdx.y * blockDim.x + threadIdx.x - lane); j0 < ldp;
         j0 += 4 * gridDim.y * blockDim.x) {
        const int j = j0 + 4 * lane;
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = (c < C && j + u < n) ? xc[j + u] : 0.0;
        int ev = e;
        if (S == 7) {
            unsigned long long m = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const unsigned long long a = abs_bits(v[u]);
                m = a > m ? a : m;
            }
            ev = oz_block_exponent(warp_max(m));
            if (lane == 0) {
                xexp[((size_t)(c / cp) * blocks + j0 / kOzBlock) * cp + c % cp] =
                    oz_pack_exponent(ev);
            }
        }
        if (j >= ldp) continue;
        const uint4 p0 = oz_pack_pair<S>(oz_biased_any<S>(v[0], ev), oz_biased_any<S>(v[1], ev));
        const uint4 p1 = oz_pack_pair<S>(oz_biased_any<S>(v[2], ev), oz_biased_any<S>(v[3], ev));
#pragma unroll
        for (int s = 0; s < S; ++s) {
            row[(size_t)s * stride + j / 4] =
                make_uint2(oz_slice_pair<S>(p0, s), oz_slice_pair<S>(p1, s));
        }
    }
    pdl_trigger();
}

// What the consumers of the partials need.
struct Partials {
    const double *P;
    const int *rowexp;
    const int *colexp;
    int n, cp, tiles, periods, maxslots, out;  // out: OzSplit::kOut
    int scaled;  // S = 7: the partials are values of Delta X
    long long items, G;
    // FP64 FMAs: the partials are `maxslots` n x C blocks of H X
    int fma, C;
    const int *err;  // set by a product whose bounded wait gave up: its results are NaN
};

// Number of partials of column c's group in a tile.
__device__ __forceinline__ int slots_of(const Partials &p, int c, int tile)
{
    if (p.fma) return p.maxslots;
    if (tile >= p.tiles) return 0;
    const long long gt = (long long)(c / p.cp) * p.tiles + tile;
    return (int)(owner_of(gt * p.periods + p.periods - 1, p.items, p.G) -
                 owner_of(gt * p.periods, p.items, p.G)) +
           1;
}

// (Delta X)_ic from its `slots` partials, in their fixed order (finite row
// and column).
__device__ __forceinline__ double delta_entry(const Partials &p, int i, int c, int slots, int ei,
                                              int fc)
{
    const int tile = i / kBM;
    const int grp = c / p.cp;
    const size_t gt = (size_t)grp * p.tiles + tile;
    const double *q = p.P + ((size_t)(gt * p.maxslots) * p.cp + (c - grp * p.cp)) * kBM +
                      (i - tile * kBM);
    const size_t stride = (size_t)p.cp * kBM;
    double s = 0.0;
#pragma unroll 4
    for (int u = 0; u < slots; ++u) s += q[u * stride];
    return p.scaled ? s : scale2(s, ei + fc + p.out);
}

// (H X)_ic from the K slices of an FP64 FMA product, in order.
__device__ __forceinline__ double fma_entry(const Partials &p, int i, int c)
{
    const size_t stride = (size_t)p.n * p.C;
    const double *q = p.P + (size_t)i + (size_t)c * p.n;
    double s = 0.0;
#pragma unroll 4
    for (int u = 0; u < p.maxslots; ++u) s += q[u * stride];
    return s;
}

constexpr int kFinishRows = 256;  // rows of one column a finish block covers

// Y[:, c] = (Delta X)[:, c] + d_i X[:, c]; NaN where the row of Delta or the
// column of X is not finite, or with H given (row i of H: H[i + l n]) the
// FP64 sum over that row, whose Inf / NaN follow the operands'.
__global__ void __launch_bounds__(kFinishRows)
oz_finish_kernel(const __grid_constant__ Partials p, const double *__restrict__ H,
                 const double *__restrict__ d, const double *__restrict__ X, long long ldx,
                 int row_blocks, double *__restrict__ Y, long long ldy)
{
    constexpr int kTiles = kFinishRows / kBM;
    __shared__ int slots[kTiles];
    const int c = blockIdx.x / row_blocks;
    const int row0 = (blockIdx.x % row_blocks) * kFinishRows;
    const int i = row0 + threadIdx.x;
    if (threadIdx.x < kTiles) slots[threadIdx.x] = slots_of(p, c, row0 / kBM + threadIdx.x);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    if (i >= p.n) return;
    const int ei = p.rowexp[i], fc = p.colexp[c];
    double y;
    if (*p.err != 0) {
        y = NAN;
    } else if (ei == kOzNonFinite || fc == kOzNonFinite) {
        y = NAN;
        if (H != nullptr) {
            y = 0.0;
            for (int l = 0; l < p.n; ++l) {
                const double h = H[(size_t)i + (size_t)l * p.n];
                if (l != i) y = fma(h, X[(size_t)l + (size_t)c * ldx], y);
            }
        }
    } else {
        y = delta_entry(p, i, c, slots[threadIdx.x / kBM], ei, fc);
    }
    if (d != nullptr) y = fma(d[i], X[(size_t)i + (size_t)c * ldx], y);
    Y[(size_t)i + (size_t)c * ldy] = y;
}

// The IPT map from the partials of Delta X:
//   c_j = (Delta X)_jj,  X'_ij = ((Delta X)_ij - X_ij c_j) g_ij,  X'_jj = 1
// (DIVIDE, the ACX map: divided by d_j - d_i, 0 where that is zero, as
// acx_cuda.cu:109-172 rounds it; 1.5 % of a call at n = 4096, k = 16),
// (IPT_C_GPU/src/ipt_cuda.cu:1369-1443), the column maxima of X' and with
// want_norms ||X' - X||_F, ||X||_F (ipt_cuda.cu:1457-1467,1663-1688); with
// resid_part also the block's part of ||(H X)_c - X_c (H X)_cc||^2 (ACX).  A
// row of H or column of X that is not finite takes the FP64 sums the map is
// defined by, so Inf and NaN travel as there.  The partials of an FP64 FMA
// product hold H X: the diagonal's part is taken off here.
//
// A block of 8 warps takes 256 R rows of one column, R per thread; a ninth
// warp forms c_j while the others load.  With R = 4 the shuffle sums of the
// norms (10 FP64 instructions per warp, each holding its partition's FP64
// pipe for 64 cycles) are shared by four rows; R = 1 while the blocks of
// R = 4 would not fill the chip.
// n = 8192, k = 32: 13 us per step together with the digit pass of X.
constexpr int kUpdateThreads = 256;

template <int R, bool RESID, bool DIVIDE>
__global__ void __launch_bounds__(kUpdateThreads + 32)
oz_update_kernel(const __grid_constant__ Partials p, const double *__restrict__ H,
                 const double *__restrict__ d, const double *__restrict__ g,
                 const double *__restrict__ X, double *__restrict__ Xn,
                 unsigned long long *__restrict__ colmax_next, int row_blocks, int want_norms,
                 int defer_norms, double2 *partials, unsigned int *counter, double *norms,
                 double *__restrict__ resid_part)
{
    constexpr int kRows = kUpdateThreads * R;
    constexpr int kTiles = kRows / kBM;
    __shared__ int slots[kTiles + 1];
    __shared__ double cj_sh;
    const int c = blockIdx.x / row_blocks;
    const int row0 = (blockIdx.x % row_blocks) * kRows;
    const int n = p.n;
    const int t = (int)threadIdx.x;
    if (t <= kTiles) slots[t] = slots_of(p, c, t < kTiles ? row0 / kBM + t : c / kBM);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const double *xc = X + (size_t)c * n;
    const int fc = p.fma ? 0 : p.colexp[c];
    // (H X)_rc - d_r X_rc by the plain FP64 sum
    auto direct = [&](int r) {
        double y = 0.0;
        for (int l = 0; l < n; ++l) y = fma(H[(size_t)r + (size_t)l * n], xc[l], y);
        return y - d[r] * xc[r];
    };
    // a product that failed gives NaN, not a sum over its NaN block per entry
    const bool failed = *p.err != 0;
    auto delta = [&](int r, int count) {
        if (failed) return (double)NAN;
        if (p.fma) return fma(-d[r], xc[r], fma_entry(p, r, c));
        const int er = p.rowexp[r];
        return (er == kOzNonFinite || fc == kOzNonFinite) ? direct(r)
                                                          : delta_entry(p, r, c, count, er, fc);
    };
    double y[R], x[R], gi[R];
    if (t < kUpdateThreads) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int i = row0 + q * kUpdateThreads + t;
            y[q] = x[q] = gi[q] = 0.0;
            if (i < n) {
                x[q] = xc[i];
                gi[q] = DIVIDE ? d[c] - d[i] : g[(size_t)i + (size_t)c * n];
                y[q] = delta(i, slots[(q * kUpdateThreads + t) / kBM]);
            }
        }
    } else if (t == kUpdateThreads) {
        cj_sh = delta(c, slots[kTiles]);
    }
    __syncthreads();
    const double cj = cj_sh;
    double dsq = 0.0, xsq = 0.0, rsq = 0.0;
    unsigned long long m = 0;
    const double hcc = RESID ? fma(d[c], xc[c], cj) : 0.0;  // (H X)_cc
    if (t < kUpdateThreads) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int i = row0 + q * kUpdateThreads + t;
            if (i < n) {
                if (RESID) {
                    const double r = fma(x[q], d[i] - hcc, y[q]);
                    rsq = fma(r, r, rsq);
                }
                double out = 1.0;
                if (i != c) {
                    out = fma(-x[q], cj, y[q]);
                    if (!DIVIDE) out *= gi[q];
                    else out = fabs(gi[q]) <= DBL_EPSILON ? 0.0 : out / gi[q];
                }
                if (failed) out = NAN;
                Xn[(size_t)i + (size_t)c * n] = out;
                const unsigned long long a = abs_bits(out);
                m = a > m ? a : m;
                if (want_norms) {
                    const double diff = out - x[q];
                    dsq = fma(diff, diff, dsq);
                    xsq = fma(x[q], x[q], xsq);
                }
            }
        }
    }
    if (!p.fma) {
        m = warp_max(m);
        if ((t & 31) == 0 && m != 0) atomicMax(colmax_next + c, m);
    }
    if (RESID) {
        const double2 r = block_sum2(rsq, 0.0);
        if (t == 0) resid_part[blockIdx.x] = r.x;
    }
    if (!want_norms) return;
    const double2 sq = block_sum2(dsq, xsq);
    if (!defer_norms) {
        grid_finish_norms2(sq, partials, counter, norms);
    } else if (t == 0) {
        partials[blockIdx.x] = sq;
    }
}

__global__ void gap_reciprocals_kernel(const double *__restrict__ d, int n, int k,
                                       double *__restrict__ g)
{
    const int j = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double gap = d[j] - d[i];
    g[(size_t)i + (size_t)j * n] = (isfinite(gap) && gap != 0.0) ? 1.0 / gap : NAN;
}

// Maxima of |H_il| (l != i) over the blocks of kOzBlock columns of each row of
// a column-major H, as bit patterns ([block][row]), and its diagonal: 256 rows x `cols` columns per block, two neighbouring rows per
// thread (16-byte loads when n is even and H aligned), eight columns in flight.
constexpr int kScanThreads = 128;
constexpr int kScanCols = 64;     // columns of a block, fewer (a power of two)
constexpr int kScanMinCols = 8;  // while the grid is small: n = 1024 16.7 -> 7.4 us

template <bool VEC>
__global__ void __launch_bounds__(kScanThreads)
oz_rowmax_kernel(const double *__restrict__ H, int n, int cols,
                 unsigned long long *__restrict__ rowmax, double *__restrict__ diag)
{
    const int i = (blockIdx.y * kScanThreads + threadIdx.x) * 2;
    if (i >= n) return;
    const int l0 = blockIdx.x * cols;
    const int l1 = min(n, l0 + cols);
    unsigned long long m0 = 0, m1 = 0;
    for (int l = l0; l < l1; l += 8) {
        double v0[8], v1[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const double *h = H + (size_t)(l + u) * n + i;
            v0[u] = v1[u] = 0.0;
            if (l + u < l1) {
                if (VEC) {
                    const double2 w = __ldcs(reinterpret_cast<const double2 *>(h));
                    v0[u] = w.x;
                    v1[u] = w.y;
                } else {
                    v0[u] = __ldcs(h);
                    if (i + 1 < n) v1[u] = __ldcs(h + 1);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const unsigned long long a0 = abs_bits(v0[u]), a1 = abs_bits(v1[u]);
            if (l + u == i) {
                if (diag != nullptr) diag[i] = v0[u];
            } else {
                m0 = a0 > m0 ? a0 : m0;
            }
            if (l + u == i + 1) {
                if (diag != nullptr && l + u < l1) diag[i + 1] = v1[u];
            } else {
                m1 = a1 > m1 ? a1 : m1;
            }
        }
    }
    unsigned long long *out = rowmax + (size_t)(l0 / kOzBlock) * n + i;
    if (m0 != 0) atomicMax(out, m0);
    if (m1 != 0 && i + 1 < n) atomicMax(out + 1, m1);
}

// Exponents of the rows and of their blocks: 32 rows per block, eight threads
// each.
__global__ void __launch_bounds__(256)
oz_rowexp_kernel(const unsigned long long *__restrict__ rowmax, int n, int blocks,
                 int *__restrict__ rowexp, uint16_t *__restrict__ blockexp)
{
    __shared__ unsigned long long part[8][32];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * 32 + lane;
    unsigned long long m = 0;
    if (i < n) {
#pragma unroll 4
        for (int b = g; b < blocks; b += 8) {
            const unsigned long long a = rowmax[(size_t)b * n + i];
            m = a > m ? a : m;
            blockexp[(size_t)b * n + i] = oz_pack_exponent(oz_block_exponent(a));
        }
    }
    part[g][lane] = m;
    __syncthreads();
    if (g != 0 || i >= n) return;
    for (int q = 1; q < 8; ++q) m = part[q][lane] > m ? part[q][lane] : m;
    rowexp[i] = oz_exponent(m);
}

// Digit words of Delta from H (words may be null): a block of threads takes
// `stages` K stages (1 or those of a kOzBlock, while that leaves enough blocks)
// of a row tile.  Lanes run along rows (coalesced reads of H); the 32 KB of a
// stage are put together in shared memory in their final order and written as
// they lie.  S = 7 counts the entries far below their block's largest,
// below[block][row], and sets *wide where a count passes oz_range_limit.
constexpr int kWordThreads = 512;
constexpr int kBlockStages = kOzBlock / kStageK;

template <int S>
__global__ void __launch_bounds__(kWordThreads)
oz_words_kernel(const double *__restrict__ H, int n, int nst, int stages,
                const int *__restrict__ rowexp, const uint16_t *__restrict__ blockexp,
                int *__restrict__ below, int *__restrict__ wide, uint4 *__restrict__ words)
{
    __shared__ uint4 img[kRawBytes / 16];
    __shared__ int count[kBM];
    const int t = (int)threadIdx.x;
    const int r = t & 127;
    const int g = t >> 7;
    const int row = blockIdx.y * kBM + r;
    const int block = blockIdx.x * stages / kBlockStages;
    int e = S == 7 ? kOzZeroExp : kOzNonFinite;
    if (row < n) e = S == 7 ? oz_unpack_exponent(blockexp[(size_t)block * n + row]) : rowexp[row];
    int far = 0;
    const int last = min((int)(blockIdx.x + 1) * stages, nst);
    for (int st = blockIdx.x * stages; st < last; ++st) {
        const int l0 = st * kStageK + 8 * g;
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int l = l0 + u;
            v[u] = (row < n && l < n) ? __ldcs(H + (size_t)l * n + row) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (l0 + u == row) v[u] = 0.0;
            else if (S == 7 && l0 + u < n && oz_far_below(v[u], e)) ++far;
        }
        if (words == nullptr) continue;
        __syncthreads();  // the stage before has been written
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            img[r * 16 + ((4 * g + p) ^ (r & 7))] =
                oz_pack_pair<S>(oz_biased_any<S>(v[2 * p], e), oz_biased_any<S>(v[2 * p + 1], e));
        }
        __syncthreads();
        uint4 *dst = words + ((size_t)blockIdx.y * nst + st) * (kRawBytes / 16);
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[q * kWordThreads + t] = img[q * kWordThreads + t];
    }
    if (S != 7) return;
    if (g == 0) count[r] = 0;
    __syncthreads();
    if (far != 0) atomicAdd(count + r, far);
    __syncthreads();
    if (g != 0 || count[r] == 0) return;
    int total = count[r];
    if (stages < kBlockStages) total += atomicAdd(below + (size_t)block * n + row, total);
    if (total > oz_range_limit(min(kOzBlock, n - block * kOzBlock), n)) *wide = 1;
}

}  // namespace oz

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
void OzMatrix::reference(const double *H_, int n_)
{
    H = H_;
    n = n_;
}

int OzMatrix::init_storage(int n_, cudaStream_t s)
{
    n = n_;
    nst = (n + oz::kStageK - 1) / oz::kStageK;
    blocks = (n + kOzBlock - 1) / kOzBlock;
    words_slices = 0;
    return rowexp.alloc((size_t)n, s);
}

int OzMatrix::alloc_words(int slices, cudaStream_t s)
{
    const size_t blocks = (size_t)((n + oz::kBM - 1) / oz::kBM) * nst;
    IPTGB_CHECK(words.alloc(blocks * (oz::kRawBytes / 16), s));
    words_slices = slices;
    return IPT_CUDA_SUCCESS;
}

namespace {
// the matrices of this thread whose words may be taken back
thread_local OzMatrix *t_held = nullptr;

// A thread has one matrix at a time between build_words() and settle().
int *make_answer()
{
    void *p = nullptr;
    if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return static_cast<int *>(p);
}
}  // namespace

bool reclaim_memory(cudaStream_t s)
{
    bool any = false;
    for (OzMatrix *m = t_held; m != nullptr; m = m->held_before) any = m->drop_words(s) || any;
    return any;
}

bool OzMatrix::drop_words(cudaStream_t s)
{
    if (words.ptr == nullptr) return false;
    const cudaStream_t owner = words.stream;
    words.release();
    words_slices = 0;
    // memory freed on one stream serves another one once that has got there
    if (owner != s) cudaStreamSynchronize(owner);
    return true;
}

OzMatrix::~OzMatrix()
{
    // (an error before settle(): the copy into the thread's slot is still due)
    if (answer != nullptr) cudaStreamSynchronize(rowexp.stream);
    if (!listed) return;
    for (OzMatrix **p = &t_held; *p != nullptr; p = &(*p)->held_before) {
        if (*p != this) continue;
        *p = held_before;
        break;
    }
}

int OzMatrix::build_words(int slices, cudaStream_t s)
{
    const size_t tiles = (size_t)(n + oz::kBM - 1) / oz::kBM;
    const size_t most = (size_t)env_int("IPT_GB300_WORDS_MAX_MB", kMaxWordMb) << 20;
    if (tiles * nst * oz::kRawBytes <= most && alloc_words(slices, s) != IPT_CUDA_SUCCESS) {
        cudaGetLastError();  // not enough memory: the product reads H itself
        words_slices = 0;
    }
    if (!listed) {
        held_before = t_held;
        t_held = this;
        listed = true;
    }
    DeviceBuffer<int> below;  // counts, and the flag behind them
    // a block of threads per kOzBlock counts without atomics in memory
    const int stages = (long long)tiles * blocks >= 4 * device_sm_count() ? oz::kBlockStages : 1;
    const size_t counts = stages == 1 ? (size_t)blocks * n : 0;
    if (slices == 7) {
        IPTGB_CHECK(below.alloc(counts + 1, s));
        IPTGB_CUDA(cudaMemsetAsync(below.ptr, 0, (counts + 1) * sizeof(int), s));
    } else if (words_slices == 0) {
        return IPT_CUDA_SUCCESS;
    }
    auto kernel = slices == 7 ? oz::oz_words_kernel<7> : oz::oz_words_kernel<6>;
    kernel<<<dim3((unsigned)((nst + stages - 1) / stages), (unsigned)tiles), oz::kWordThreads, 0,
             s>>>(H, n, nst, stages, rowexp.ptr, blockexp.ptr, below.ptr, below.ptr + counts,
                  words.ptr);
    IPTGB_LAUNCH();
    if (slices != 7) return IPT_CUDA_SUCCESS;
    answer = ThreadSlots<int>::mine(make_answer);
    if (answer == nullptr) return IPT_CUDA_ALLOCATION_FAILED;
    IPTGB_CUDA(cudaMemcpyAsync(answer, below.ptr + counts, sizeof(int), cudaMemcpyDeviceToHost, s));
    return IPT_CUDA_SUCCESS;
}

// The setup of the first step is queued between build_words() and this: the
// wait then costs a small solve (n = 1024) 10 us less.
int OzMatrix::settle(cudaStream_t s)
{
    if (answer == nullptr) return IPT_CUDA_SUCCESS;
    IPTGB_CUDA(cudaStreamSynchronize(s));
    wide = *answer != 0;
    answer = nullptr;
    if (wide) {
        words.release();
        words_slices = 0;
    }
    return IPT_CUDA_SUCCESS;
}

int OzMatrix::scan_rows(const double *H_, int n_, double *diag, cudaStream_t s)
{
    IPTGB_CHECK(init_storage(n_, s));
    H = H_;
    DeviceBuffer<unsigned long long> rm;
    const size_t maxima = (size_t)blocks * n;
    IPTGB_CHECK(blockexp.alloc(maxima, s));
    IPTGB_CHECK(rm.alloc(maxima, s));
    IPTGB_CUDA(cudaMemsetAsync(rm.ptr, 0, maxima * sizeof(unsigned long long), s));
    const int rows = 2 * oz::kScanThreads;
    const int row_blocks = (n + rows - 1) / rows;
    int cols = oz::kScanCols;
    const int enough = 3 * device_sm_count();
    while (cols > oz::kScanMinCols && (long long)((n + cols - 1) / cols) * row_blocks < enough) {
        cols /= 2;
    }
    const dim3 grid((n + cols - 1) / cols, row_blocks);
    const bool vec = n % 2 == 0 && (reinterpret_cast<uintptr_t>(H) & 15) == 0;
    auto scan = vec ? oz::oz_rowmax_kernel<true> : oz::oz_rowmax_kernel<false>;
    scan<<<grid, oz::kScanThreads, 0, s>>>(H, n, cols, rm.ptr, diag);
    IPTGB_LAUNCH();
    oz::oz_rowexp_kernel<<<(n + 31) / 32, 256, 0, s>>>(rm.ptr, n, blocks, rowexp.ptr,
                                                       blockexp.ptr);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

namespace {

// Columns per group: up to 64 for the 48-bit split (its 6 level accumulators
// then fill TMEM), 32 for the 56-bit split (8 levels, two accumulator sets).
int group_cols(int slices, int C)
{
    const int most = slices == 7 ? 32 : 64;
    return std::min(most, (C + 15) / 16 * 16);
}

template <int S, int CP, int MODE>
int launch_product(const CUtensorMap &mapB, const oz::Params &prm, int grid, double *P, int *err,
                   cudaStream_t s)
{
    auto kfn = oz::oz_product_kernel<S, CP, MODE>;
    constexpr size_t smem = oz::Layout<S, CP>::kSmem;
    IPTGB_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch_pdl(kfn, dim3(grid), dim3(oz::kThreads), smem, s, mapB, prm, P, err);
}

template <int MODE>
int launch_product_for(int slices, int cp, const CUtensorMap &mapB, const oz::Params &prm, int grid,
                       double *P, int *err, cudaStream_t s)
{
    if (slices == 7) {
        return cp == 16 ? launch_product<7, 16, MODE>(mapB, prm, grid, P, err, s)
                        : launch_product<7, 32, MODE>(mapB, prm, grid, P, err, s);
    }
    switch (cp) {
    case 16: return launch_product<6, 16, MODE>(mapB, prm, grid, P, err, s);
    case 32: return launch_product<6, 32, MODE>(mapB, prm, grid, P, err, s);
    case 48: return launch_product<6, 48, MODE>(mapB, prm, grid, P, err, s);
    default: return launch_product<6, 64, MODE>(mapB, prm, grid, P, err, s);
    }
}

int make_tile_map(CUtensorMap *map, CUtensorMapDataType dt, int esize, const void *base,
                  size_t inner, size_t outer, int box_inner, int box_outer, CUtensorMapSwizzle sw)
{
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return IPT_CUDA_CUDA_ERROR;
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
    cuuint64_t strides[1] = {(cuuint64_t)inner * esize};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, dt, 2, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        fprintf(stderr, "ipt_gb300: cuTensorMapEncodeTiled failed (%d)\n", (int)r);
        return IPT_CUDA_CUDA_ERROR;
    }
    return IPT_CUDA_SUCCESS;
}

}  // namespace

int OzProduct::bind(const OzMatrix *matrix, const double *diag, int digit_slices,
                    cudaStream_t stream)
{
    if (m != matrix || slices != digit_slices) sh = OzShape();
    m = matrix;
    d = diag;
    s = stream;
    slices = digit_slices;
    sms = device_sm_count();
    const int limit = env_int("IPT_GB300_SPIN_LIMIT", 0);
    spin = limit > 0 ? limit : tc::kSpinLimit;
    if (err.ptr == nullptr) {
        IPTGB_CHECK(err.alloc(1, s));
        IPTGB_CUDA(cudaMemsetAsync(err.ptr, 0, sizeof(int), s));
    }
    return IPT_CUDA_SUCCESS;
}

int OzProduct::shape_for(int C)
{
    if (sh.C == C && sh.n == m->n) return IPT_CUDA_SUCCESS;
    const int n = m->n;
    OzShape q;
    q.n = n;
    q.C = C;
    if (slices == 0) {
        q.maxslots = dense64_split_for(n, C, sms);
        const size_t need = (size_t)q.maxslots * n * C;
        if (P.count < need) IPTGB_CHECK(P.alloc(need, s));
        sh = q;
        return IPT_CUDA_SUCCESS;
    }
    q.cp = group_cols(slices, C);
    q.groups = (C + q.cp - 1) / q.cp;
    q.tiles = (n + oz::kBM - 1) / oz::kBM;
    q.ldp = (n + 63) / 64 * 64;
    // Items of kOzPeriod K elements, or (56-bit split, whose sums do not depend
    // on it) half or a quarter of that while it shortens the longest CTA: a
    // matrix of a few tiles then spreads over more SMs.  An item's drain takes
    // about as long as three stages (6400 cycles) beside the MMAs of the next.
    const int nst = (n + oz::kStageK - 1) / oz::kStageK;
    long long best = LLONG_MAX;
    for (int spp = oz::kMaxStagesPerItem; spp >= (slices == 7 ? 1 : oz::kMaxStagesPerItem);
         spp /= 2) {
        const int periods = (nst + spp - 1) / spp;
        const long long items = (long long)q.groups * q.tiles * periods;
        const long long longest =
            (items + sms - 1) / sms * (slices == 7 ? std::max(spp, 3) : spp);
        if (longest >= best) continue;
        best = longest;
        q.spp = spp;
        q.periods = periods;
        q.items = items;
    }
    q.grid = (int)std::min<long long>(sms, q.items);
    q.maxslots = 1;
    for (long long t = 0; t < (long long)q.groups * q.tiles; ++t) {
        const long long f = tc::owner_of(t * q.periods, q.items, q.grid);
        const long long l = tc::owner_of(t * q.periods + q.periods - 1, q.items, q.grid);
        q.maxslots = std::max(q.maxslots, (int)(l - f + 1));
    }
    const size_t rows = (size_t)q.groups * slices * q.cp;
    const size_t bneed = rows * q.ldp;
    const size_t pneed = (size_t)q.groups * q.tiles * q.maxslots * q.cp * oz::kBM;
    const size_t cneed = (size_t)q.groups * q.cp;
    if (B.count < bneed) IPTGB_CHECK(B.alloc(bneed, s));
    if (colexp.count < cneed) IPTGB_CHECK(colexp.alloc(cneed, s));
    if (slices == 7 && xexp.count < cneed * m->blocks) {
        IPTGB_CHECK(xexp.alloc(cneed * m->blocks, s));
    }
    if (colmax.count < 2 * cneed) IPTGB_CHECK(colmax.alloc(2 * cneed, s));
    if (P.count < pneed) IPTGB_CHECK(P.alloc(pneed, s));
    cur = 0;
    // digits: box of 64 bytes of K x the rows of a group (half of them when
    // they exceed the 256 rows a box may have)
    const int box_rows = slices * q.cp <= 256 ? slices * q.cp : slices / 2 * q.cp;
    IPTGB_CHECK(make_tile_map(&mapB, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, B.ptr, q.ldp, rows,
                              oz::kStageK, box_rows, CU_TENSOR_MAP_SWIZZLE_64B));
    sh = q;
    return IPT_CUDA_SUCCESS;
}

// B slices of X from the maxima of set `cur` (clearing the other set), then
// the partials of Delta X.
int OzProduct::slice_and_multiply(const double *X, long long ldx, int clear_other)
{
    const OzShape &q = sh;
    const size_t set = (size_t)q.groups * q.cp;
    const int pc = q.groups * q.cp;
    const int ychunks = std::max(1, std::min((q.ldp + 1023) / 1024, (8 * sms + pc - 1) / pc));
    auto slice = slices == 7 ? oz::oz_slice_x_kernel<7> : oz::oz_slice_x_kernel<6>;
    const oz::PendingNorms norms = {pending_parts, pending_count, pending_out};
    IPTGB_CHECK(launch_pdl(slice, dim3(pc + (pending_count > 0 ? 1 : 0), ychunks), dim3(256), 0, s,
                           X, ldx, q.n, q.C, q.cp, q.ldp,
                           (const unsigned long long *)(colmax.ptr + cur * set),
                           clear_other ? colmax.ptr + (1 - cur) * set : nullptr, B.ptr,
                           colexp.ptr, xexp.ptr, m->blocks, norms));
    pending_count = 0;
    oz::Params prm = {};
    prm.H = m->H;
    prm.words = m->words.ptr;
    prm.rowexp = m->rowexp.ptr;
    prm.blockexp = m->blockexp.ptr;
    prm.xexp = reinterpret_cast<const uint32_t *>(xexp.ptr);
    prm.blocks = m->blocks;
    prm.n = q.n;
    prm.groups = q.groups;
    prm.tiles = q.tiles;
    prm.periods = q.periods;
    prm.spp = q.spp;
    prm.nstages = m->nst;
    prm.items = q.items;
    prm.maxslots = q.maxslots;
    prm.stream_h = (size_t)q.n * q.n * sizeof(double) > oz::kL2ResidentBytes;
    prm.b_loads = slices * q.cp <= 256 ? 1 : 2;
    prm.b_bytes = (uint32_t)(slices * q.cp * 64);
    prm.spin = spin;
    auto launch = m->words_slices == slices ? launch_product_for<oz::kWords>
                                            : launch_product_for<oz::kRows>;
    return launch(slices, q.cp, mapB, prm, q.grid, P.ptr, err.ptr, s);
}

oz::Partials OzProduct::partials() const
{
    oz::Partials p;
    p.P = P.ptr;
    p.fma = slices == 0;
    p.C = sh.C;
    p.rowexp = m->rowexp.ptr;
    p.colexp = colexp.ptr;
    p.n = sh.n;
    p.cp = sh.cp;
    p.tiles = sh.tiles;
    p.periods = sh.periods;
    p.maxslots = sh.maxslots;
    p.out = OzSplit<6>::kOut;
    p.scaled = slices == 7;
    p.items = sh.items;
    p.G = sh.grid;
    p.err = err.ptr;
    return p;
}

int OzProduct::scan_columns(const double *X, long long ldx)
{
    const size_t set = (size_t)sh.groups * sh.cp;
    IPTGB_CUDA(cudaMemsetAsync(colmax.ptr + cur * set, 0, set * sizeof(unsigned long long), s));
    const int ychunks = std::max(1, std::min((sh.n + 2047) / 2048, (4 * sms + sh.C - 1) / sh.C));
    return launch_pdl(oz::oz_colmax_kernel, dim3(sh.C, ychunks), dim3(256), 0, s, X, ldx, sh.n,
                      colmax.ptr + cur * set);
}

int OzProduct::apply(const double *X, long long ldx, int C, double *Y, long long ldy)
{
    if (C <= 0) return IPT_CUDA_SUCCESS;
    IPTGB_CHECK(shape_for(C));
    IPTGB_CHECK(scan_columns(X, ldx));
    IPTGB_CHECK(slice_and_multiply(X, ldx, 0));
    const int row_blocks = (sh.n + oz::kFinishRows - 1) / oz::kFinishRows;
    return launch_pdl(oz::oz_finish_kernel, dim3((unsigned)((long long)row_blocks * C)),
                      dim3(oz::kFinishRows), 0, s, partials(),
                      slices == 7 ? m->H : (const double *)nullptr, d, X, ldx, row_blocks, Y, ldy);
}

int OzProduct::begin(const double *X, int C)
{
    IPTGB_CHECK(shape_for(C));
    return slices == 0 ? IPT_CUDA_SUCCESS : scan_columns(X, sh.n);
}

int OzProduct::update_row_blocks(int n, int C, int sms, bool *wide)
{
    const int r1 = (n + oz::kUpdateThreads - 1) / oz::kUpdateThreads;
    *wide = (long long)((r1 + 3) / 4) * C >= sms;
    return *wide ? (r1 + 3) / 4 : r1;
}

int OzProduct::flush_norms()
{
    if (pending_count == 0) return IPT_CUDA_SUCCESS;
    const oz::PendingNorms norms = {pending_parts, pending_count, pending_out};
    pending_count = 0;
    return launch_pdl(oz::oz_norms_kernel, dim3(1), dim3(256), 0, s, norms);
}

int OzProduct::step(const double *X, const double *g, double *Xn, int want_norms, NormScratch *ns,
                    double *resid_part, bool defer_norms)
{
    bool wide = false;
    const int row_blocks = update_row_blocks(sh.n, sh.C, sms, &wide);
    const long long grid = (long long)row_blocks * sh.C;
    if (want_norms && grid > ns->capacity) return IPT_CUDA_INVALID_ARGUMENT;
    const size_t set = (size_t)sh.groups * sh.cp;
    {
        KernelTimerScope timer(kProfFp64Product, s);
        if (slices == 0) {
            IPTGB_CHECK(launch_dense64_partial(m->H, sh.n, sh.n, X, sh.n, sh.C, P.ptr,
                                               sh.maxslots, s));
            defer_norms = false;  // (there is no digit pass to finish them)
        } else {
            IPTGB_CHECK(slice_and_multiply(X, sh.n, 1));
        }
    }
    KernelTimerScope timer(kProfFp64Update, s);
    auto update =
        g != nullptr ? (wide ? oz::oz_update_kernel<4, false, false>
                             : oz::oz_update_kernel<1, false, false>)
        : resid_part == nullptr ? (wide ? oz::oz_update_kernel<4, false, true>
                                        : oz::oz_update_kernel<1, false, true>)
                                : (wide ? oz::oz_update_kernel<4, true, true>
                                        : oz::oz_update_kernel<1, true, true>);
    if (g != nullptr && resid_part != nullptr) return IPT_CUDA_INVALID_ARGUMENT;
    IPTGB_CHECK(launch_pdl(update,
                           dim3((unsigned)grid), dim3(oz::kUpdateThreads + 32), 0, s, partials(),
                           m->H, d, g, X, Xn, colmax.ptr + (1 - cur) * set, row_blocks,
                           want_norms, defer_norms ? 1 : 0, ns->partials, ns->counter, ns->norms,
                           resid_part));
    if (want_norms && defer_norms) {
        pending_parts = ns->partials;
        pending_count = (int)grid;
        pending_out = ns->norms;
    }
    cur = 1 - cur;
    return IPT_CUDA_SUCCESS;
}

int OzProduct::check()
{
    if (err.ptr == nullptr || slices == 0) return IPT_CUDA_SUCCESS;
    int code = 0;
    IPTGB_CHECK(read_error(&code));
    if (code == 0) return IPT_CUDA_SUCCESS;
    fprintf(stderr, "ipt_gb300: FP64-accurate product: pipeline wait %d gave up\n", code);
    return IPT_CUDA_CUDA_ERROR;
}

int OzProduct::read_error(int *host_err)
{
    IPTGB_CUDA(cudaMemcpyAsync(host_err, err.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    IPTGB_CUDA(cudaStreamSynchronize(s));
    return IPT_CUDA_SUCCESS;
}

bool fp64_fma_wanted()
{
    const char *ap = getenv("IPT_GB300_ACCURATE_PRODUCT");
    return env_flag("IPT_GB300_FP64_DFMA", 0) != 0 || (ap != nullptr && strcmp(ap, "fp64") == 0);
}

int launch_gap_reciprocals(const double *d, int n, int k, double *g, cudaStream_t s)
{
    oz::gap_reciprocals_kernel<<<dim3((n + kThreads - 1) / kThreads, k), kThreads, 0, s>>>(d, n, k,
                                                                                          g);
    IPTGB_LAUNCH();
    return IPT_CUDA_SUCCESS;
}

}  // namespace iptgb

// ---------------------------------------------------------------------------
// Exported entry points (include/ipt_block.h)
// ---------------------------------------------------------------------------
#define IPT_API extern "C" __attribute__((visibility("default")))

IPT_API int ipt_block_accurate_product(const double *d_H, int n, const double *d_X, int c,
                                       double *d_Y, void *stream)
{
    using namespace iptgb;
    if (d_H == nullptr || d_X == nullptr || d_Y == nullptr || n <= 0 || c <= 0 ||
        (size_t)n * (size_t)c > (size_t)INT_MAX) {
        return IPT_CUDA_INVALID_ARGUMENT;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DeviceBuffer<double> d;
    IPTGB_CHECK(d.alloc((size_t)n, s));
    OzMatrix matrix;
    IPTGB_CHECK(matrix.scan_rows(d_H, n, d.ptr, s));
    OzProduct prod;
    IPTGB_CHECK(prod.bind(&matrix, d.ptr, kOzSlices, s));
    IPTGB_CHECK(prod.apply(d_X, n, c, d_Y, n));
    int herr = 0;
    IPTGB_CHECK(prod.read_error(&herr));
    if (herr != 0) {
        fprintf(stderr, "ipt_gb300: accurate product: bounded wait gave up (code %d)\n", herr);
        return IPT_CUDA_CUDA_ERROR;
    }
    IPTGB_CUDA(cudaGetLastError());
    return IPT_CUDA_SUCCESS;
}

IPT_API int ipt_block_accurate_split_host(const double *values, long long count, double max_abs,
                                          int *exponent_out, int *digits_out)
{
    using namespace iptgb;
    if (count < 0 || exponent_out == nullptr || (count > 0 && (values == nullptr ||
                                                               digits_out == nullptr))) {
        return IPT_CUDA_INVALID_ARGUMENT;
    }
    uint64_t mb;
    memcpy(&mb, &max_abs, sizeof(mb));
    const int e = oz_exponent(mb & 0x7FFFFFFFFFFFFFFFULL);
    *exponent_out = e;
    for (long long i = 0; i < count; ++i) {
        int dg[kOzSlices];
        oz_digits_of(oz_fixed(values[i], e), dg);
        for (int s = 0; s < kOzSlices; ++s) digits_out[i * kOzSlices + s] = dg[s];
    }
    return IPT_CUDA_SUCCESS;
}
