// oz.cuh - operand splitting of the FP64-accurate tensor-core products
// (internal; host and device).
//
// The product Y = Delta X with FP64 operands runs on the FP16 tensor cores
// by the error-free split-operand scheme of Ozaki, Ogita, Oishi and Rump
// ("Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication and its applications", Numer. Algorithms
// 59 (2012)), in the fixed-point form that Mukunoki, Ozaki, Ogita and Imamura
// run on tensor cores ("DGEMM using Tensor Cores, and Its Accurate and
// Reproducible Versions", ISC 2020):
//
//  * every row i of Delta is scaled by 2^-e_i, e_i the smallest exponent
//    with max_j |Delta_ij| < 2^e_i, and rounded to the fixed-point integer
//    Q_ij = round(Delta_ij 2^(F - e_i)); every column c of X likewise with
//    its own exponent f_c (S = 7: every block of 128 entries of a row or
//    column has its own);
//  * Q is written in S balanced base-256 digits, Q = sum_s A_s 256^(S-1-s),
//    A_s in [-128, 127] for s > 0: small integers that FP16 holds exactly;
//  * the level sums L_l = sum_{s+t=l} A_s B_t are kept for l < V, the
//    products of lower weight are dropped.  Every level sum over kOzPeriod
//    consecutive K elements stays within 2^24, so the tensor cores' FP32
//    accumulation adds integers exactly; the accumulators are drained every
//    kOzPeriod K elements.
//
// Two instances (OzSplit<S>):
//  * S = 6, F = 48, V = 6 (the mixed solve's defect and certification
//    products): A_0 in [-256, 256]; the dropped products are each below
//    2^-47 of the fixed-point scale; drains are combined in double-float
//    arithmetic.
//  * S = 7, F = 56, V = 8, rounded toward zero (the plain FP64 path): 56 bits
//    hold every bit of a double within three binades of the largest entry of
//    its block (kOzBlock); the errors are the truncation of the operands
//    below 2^-56 of their block's scale and the dropped products, each below
//    2^-64 of the product of the scales.  Levels 0 to 5 stay within 2^24 and
//    add exactly; a level sum 6 or 7 beyond it may round by one unit, 2^-64
//    of the scale.  Drains are added as 96-bit integers at the largest scale
//    so far, cut off below 2^-72 of it.  Over one block an entry of Delta X
//    is off by up to 128 2^-54 max|Delta_il| max|X_lc|, where FP64 FMAs are
//    off by a few 2^-53 sum |Delta_il X_lc|: the same where the entries of a
//    row of Delta do not span many binades within a block.  oz_range_limit
//    is the line beyond which a matrix is multiplied in FP64 FMAs.
//
// The rounding to Q and the digit extraction use integer operations only
// (GB300 runs FP64 arithmetic at 1/64 of the FP32 rate).
#pragma once

#include <stdint.h>

namespace iptgb {

constexpr int kOzSlices = 6;      // digits per operand of the 48-bit split
constexpr int kOzPeriod = 128;    // K elements between accumulator drains
constexpr int kOzBlock = 128;     // S = 7: K elements of a row or column that share an exponent
static_assert(kOzBlock % kOzPeriod == 0, "a drain's K elements share their exponents");

// S slices: F fixed-point bits, V digit-product levels kept, the bias that
// makes the low S - 1 digits unsigned bytes and puts the top digit, as the
// FP16 bit pattern of 1536 + digit, into the 16 bits above them, and the
// product's scale: Y = 2^(e_i + f_c + kOut) * (sum of the drains).
template <int S>
struct OzSplit;
template <>
struct OzSplit<6> {
    static constexpr int kBits = 48, kLevels = 6, kOut = -16;
    static constexpr uint64_t kBias = 0x0066008080808080ULL;
};
template <>
struct OzSplit<7> {
    static constexpr int kBits = 56, kLevels = 8, kOut = -72;
    static constexpr uint64_t kBias = 0x6600808080808080ULL;
};
// Row / column exponent of a row that holds Inf or NaN: the product of that
// row (column) is NaN.
constexpr int kOzNonFinite = 0x7fffffff;
// Exponent of a block of zeros (S = 7): below every other.
constexpr int kOzZeroExp = -8192;

#if defined(__CUDACC__)
#define OZ_HD __host__ __device__ __forceinline__
#else
#define OZ_HD inline
#endif

// Smallest e with |v| < 2^e for the absolute-value bit pattern `absbits` of
// the largest |v| (0 for an all-zero row, kOzNonFinite for Inf / NaN).
OZ_HD int oz_exponent(uint64_t absbits)
{
    if (absbits == 0) return 0;
    const int E = (int)(absbits >> 52);
    if (E == 2047) return kOzNonFinite;
    if (E == 0) {
        // subnormal: absbits * 2^-1074 < 2^(p + 1 - 1074), p the top set bit
        int p = 0;
        while ((absbits >> (p + 1)) != 0) ++p;
        return p + 1 - 1074;
    }
    return E - 1022;  // 1.f * 2^(E - 1023) < 2^(E - 1022)
}

// The same for a block of kOzBlock entries.
OZ_HD int oz_block_exponent(uint64_t absbits)
{
    return absbits == 0 ? kOzZeroExp : oz_exponent(absbits);
}

// A block's exponent as the product kernel keeps it: 16 bits, biased so that a
// sum of two is positive and below 2^15.  A block that is not finite has zero
// digits, as one of zeros (its row or column is not taken from the product).
OZ_HD uint16_t oz_pack_exponent(int e)
{
    return (uint16_t)(e == kOzNonFinite ? 0 : e - kOzZeroExp);
}

OZ_HD int oz_unpack_exponent(uint16_t p)
{
    return (int)p + kOzZeroExp;
}

// Does an entry lie more than six binades below its block's largest, of
// exponent e?
OZ_HD bool oz_far_below(double v, int e)
{
    uint64_t b;
#if defined(__CUDA_ARCH__)
    b = (uint64_t)__double_as_longlong(v);
#else
    __builtin_memcpy(&b, &v, sizeof(b));
#endif
    return (int)((b >> 52) & 0x7FFu) + 6 < e + 1022;
}

// The number of off-diagonal entries of a block that may lie that far below
// (of its `count` columns, in a matrix of n): 3/8 of them, 8 more in the short
// block at the end of a longer row.  Median relative errors of the vectors'
// entries after 8 steps, k = 8, FP64 FMAs | this split: couplings N(0,1) with
// a decay of exp(-|i-j|/64), n = 1500 (28 % below in the worst block) 9e-16 |
// 6e-16; graded (d from 1 to 1e20, couplings ~ sqrt(d_i d_j)), n = 1024 (30 %)
// 8e-16 | 1e-15; beyond the line, graded 1 to 1e12, n = 300 (63 %) 4e-16 |
// 2e-14; decay exp(-|i-j|/16) (76 %) 8e-16 | 9e-14; tridiagonal: the small
// entries are lost.
OZ_HD int oz_range_limit(int count, int n)
{
    return 3 * count / 8 + (count < kOzBlock && n > kOzBlock ? 8 : 0);
}

// The F-bit fixed-point value round(v 2^(F - e)) (round half away from
// zero) of a finite v with |v| < 2^e; 0 for non-finite v.
template <int F>
OZ_HD int64_t oz_fixed_bits(double v, int e)
{
    uint64_t b;
#if defined(__CUDA_ARCH__)
    b = (uint64_t)__double_as_longlong(v);
#else
    __builtin_memcpy(&b, &v, sizeof(b));
#endif
    const bool neg = (b >> 63) != 0;
    b &= 0x7FFFFFFFFFFFFFFFULL;
    const int E = (int)(b >> 52);
    if (E == 2047 || b == 0 || e == kOzNonFinite) return 0;
    uint64_t M;
    int x;  // |v| = M * 2^x
    if (E == 0) {
        M = b;
        x = -1074;
    } else {
        M = (b & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL;
        x = E - 1075;
    }
    const int sh = e - F - x;  // Q = M * 2^-sh
    uint64_t q;
    if (sh >= 60) {
        q = 0;
    } else if (sh > 0) {
        q = (M >> sh) + ((M >> (sh - 1)) & 1ULL);
    } else {
        q = M << (-sh);  // exact: the row's largest entry is close to v
    }
    return neg ? -(int64_t)q : (int64_t)q;
}

OZ_HD int64_t oz_fixed(double v, int e)
{
    return oz_fixed_bits<OzSplit<6>::kBits>(v, e);
}

// Balanced base-256 digits of a fixed-point value: q = sum_s d[s] 256^(5-s).
OZ_HD void oz_digits_of(int64_t q, int (&d)[kOzSlices])
{
#pragma unroll
    for (int s = kOzSlices - 1; s >= 1; --s) {
        const int64_t r = ((q + 128) & 255) - 128;
        d[s] = (int)r;
        q = (q - r) >> 8;  // exact: q - r is a multiple of 256
    }
    d[0] = (int)q;
}

// Rows (columns) whose scale is below 2^kOzFastExp take the general form of
// the split; subnormal entries of all others round to zero.
constexpr int kOzFastExp = -900;

// The offset nb that oz_biased subtracts an entry's exponent field from, for
// a row of exponent e >= kOzFastExp (a non-finite row gets zero digits).
template <int S>
OZ_HD int oz_shift_base(int e)
{
    return e == kOzNonFinite ? 4096 : e + (S == 6 ? 1029 : 1022);
}

// Q + bias for an entry v of a row with shift base nb.  Adding 128 to every
// digit below the top one turns the balanced digits into the bytes of the
// sum (no carries to propagate): byte j holds digit S-1-j plus 128, the 16
// bits above the S - 1 bytes hold 0x6600 + A_0.  With M the 53-bit
// significand, one 64-bit shift of 8 M gives floor(|Q|) (S = 7), or
// t = floor(2 |Q|) and the rounded |Q| = (t + 1) >> 1 (S = 6).
template <int S>
OZ_HD uint64_t oz_biased(double v, int nb)
{
    uint64_t b;
#if defined(__CUDA_ARCH__)
    b = (uint64_t)__double_as_longlong(v);
#else
    __builtin_memcpy(&b, &v, sizeof(b));
#endif
    const uint32_t hi = (uint32_t)(b >> 32);
    const uint32_t sh = (uint32_t)(nb - (int)((hi >> 20) & 0x7FFu));
    const uint32_t n8 = sh < 63u ? sh : 63u;
    const uint64_t m8 = ((b << 3) & 0x007FFFFFFFFFFFFFULL) | 0x0080000000000000ULL;
    uint64_t q = m8 >> n8;
    if (S == 6) q = (q + 1) >> 1;
    // two's complement by the sign, and the bias: its low word takes the
    // + 1 without a carry
    const uint32_t sg = (uint32_t)((int32_t)hi >> 31);
    const uint64_t x = ((uint64_t)((uint32_t)(q >> 32) ^ sg) << 32) | ((uint32_t)q ^ sg);
    const uint32_t low = (uint32_t)OzSplit<S>::kBias + (hi >> 31);
    return x + ((OzSplit<S>::kBias & 0xFFFFFFFF00000000ULL) | low);
}

// The same for any row exponent.
template <int S>
OZ_HD uint64_t oz_biased_any(double v, int e)
{
    if (e != kOzNonFinite && e < kOzFastExp) {
        return (uint64_t)oz_fixed_bits<OzSplit<S>::kBits>(v, e) + OzSplit<S>::kBias;
    }
    return oz_biased<S>(v, oz_shift_base<S>(e));
}

// The S digits packed in a biased value.
template <int S>
OZ_HD void oz_unpack(uint64_t w, int (&d)[S])
{
#pragma unroll
    for (int s = 1; s < S; ++s) d[s] = (int)((w >> (8 * (S - 1 - s))) & 255u) - 128;
    d[0] = (int)((w >> (8 * (S - 1))) & 0xFFFFu) - 0x6600;
}

// The digits of oz_digits_of(oz_fixed(v, e)) as the kernels form them.
OZ_HD void oz_digits_fast(double v, int e, int (&d)[kOzSlices])
{
    oz_unpack<kOzSlices>(oz_biased_any<kOzSlices>(v, e), d);
}

}  // namespace iptgb

#if defined(__CUDACC__)
#include <cuda_fp16.h>

namespace iptgb {

// The digits of two neighbouring entries, from their biased values, as four
// words: x = digits S-1 and S-2 of both (bytes: entry 0, entry 1, entry 0,
// entry 1), y = digits S-3 and S-4, z = the one or two digits left, w = the
// top digits' FP16 patterns.
template <int S>
__device__ __forceinline__ uint4 oz_pack_pair(uint64_t w0, uint64_t w1)
{
    const uint32_t l0 = (uint32_t)w0, l1 = (uint32_t)w1;
    const uint32_t u0 = (uint32_t)(w0 >> 32), u1 = (uint32_t)(w1 >> 32);
    return make_uint4(__byte_perm(l0, l1, 0x5140), __byte_perm(l0, l1, 0x7362),
                      __byte_perm(u0, u1, 0x5140),
                      __byte_perm(u0, u1, S == 7 ? 0x7632 : 0x6521));
}

// FP16 digit pairs (first entry in the low half) from two bytes of a packed
// word (sel 0x4140: the low two, 0x4342: the high two): a byte u under 0x64 is
// the FP16 value 1024 + u, and subtracting 1152 leaves the digit u - 128,
// exactly; 1536 for the top digit's word.
__device__ __forceinline__ uint32_t oz_half_pair(uint32_t word, uint32_t sel)
{
    const uint32_t b = __byte_perm(word, 0x64646464u, sel);
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&b), __float2half2_rn(1152.0f));
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ uint32_t oz_top_pair(uint32_t word)
{
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&word), __float2half2_rn(1536.0f));
    return *reinterpret_cast<const uint32_t *>(&v);
}

// Digit pair of slice s from a packed pair.
template <int S>
__device__ __forceinline__ uint32_t oz_slice_pair(const uint4 &p, int s)
{
    if (s == 0) return oz_top_pair(p.w);
    const int j = S - 1 - s;  // byte of the biased value
    return oz_half_pair(j < 2 ? p.x : j < 4 ? p.y : p.z, (j & 1) != 0 ? 0x4342u : 0x4140u);
}

// Digit words of Delta: per 128-row tile and 32-element K stage one 32 KB
// block [row][16 pairs], the 16-byte pair j of row r at position j ^ (r % 8)
// (the product kernel's 16-byte shared-memory reads, lanes = rows, then meet
// every bank).  Index of the pair that holds K entry l (and l ^ 1) of `row`,
// with nst stages per row.
__host__ __device__ __forceinline__ size_t oz_word_index(int row, int l, int nst)
{
    const int r = row & 127;
    return (((size_t)(row >> 7) * nst + (l >> 5)) * 128 + r) * 16 + (((l & 31) >> 1) ^ (r & 7));
}

}  // namespace iptgb
#endif
