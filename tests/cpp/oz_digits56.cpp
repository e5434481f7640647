// Checks the 56-bit operand split of the FP64-accurate tensor-core product
// (block_ipt_gb300/csrc/oz.cuh, oz_biased_any<7>): seven digits, the top one
// in [-256, 256], the others in [-128, 127], whose value is v 2^(56 - e)
// rounded toward zero (to nearest for rows below the fast path's range), for
// scaled, full-exponent, exact, subnormal-scale, zero and non-finite rows.
// Built and run by tests/test_plain_split.py.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "oz.cuh"
using namespace iptgb;
int main() {
    std::mt19937_64 rng(11);
    long long bad = 0, n = 0;
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    for (int trial = 0; trial < 3000000; ++trial) {
        double v; int e = 0;
        const int kind = trial % 6;
        if (kind == 0) { v = u(rng); }
        else if (kind == 1) { v = std::ldexp(u(rng), -(int)(rng() % 80)); }
        else if (kind == 2) { uint64_t b = (rng() & 0x800FFFFFFFFFFFFFULL) | ((uint64_t)(rng() % 1990 + 56) << 52); std::memcpy(&v, &b, 8); int ex; std::frexp(v, &ex); e = ex + (int)(rng() % 60); if (e > 1024) e = 1024; }
        else if (kind == 3) { v = std::ldexp((double)((long long)(rng() % 512) - 256), -8 * (int)(rng() % 7) - 8); }
        else if (kind == 4) { uint64_t b = rng() % 0x000FFFFFFFFFFFFFULL; std::memcpy(&v, &b, 8); e = -1000 + (int)(rng() % 40); }
        else { v = 0.0; e = (int)(rng() % 10); }
        if (kind == 3 && std::fabs(v) >= 1.0) v = 0.5;
        int d[7];
        oz_unpack<7>(oz_biased_any<7>(v, e), d);
        long long q = 0;
        bool ok = d[0] >= -256 && d[0] <= 256;
        for (int s = 0; s < 7; ++s) { q = q * 256 + d[s]; if (s) ok = ok && d[s] >= -128 && d[s] <= 127; }
        // long double holds v 2^(56 - e) exactly
        const long double x = std::ldexp((long double)v, 56 - e);
        const long long want = e < kOzFastExp ? (long long)std::llroundl(x) : (long long)std::truncl(x);
        ok = ok && q == want;
        ++n;
        if (!ok) { if (bad < 5) printf("mismatch v=%.17g e=%d q=%lld want=%lld\n", v, e, q, want); ++bad; }
    }
    int d[7];
    oz_unpack<7>(oz_biased_any<7>(3.0, kOzNonFinite), d);
    for (int s = 0; s < 7; ++s) bad += d[s] != 0;
    printf("checked %lld mismatches %lld\n", n, bad);
    return bad != 0;
}
