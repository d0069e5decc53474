// Host check of fq_smulc, the integer-pipe product by a prepared factor (fq_soft64.h), against the
// host's IEEE product (compile with -ffp-contract=off).  Usage: soft64_factor_check <factor family> <cases
// per factor>.  Factor families: 0 step parameters, 1 random, 2 few-bit, 3 not normal or near the ends of
// the exponent range.  Prints operations, mismatches, operations that took the hardware path.
#include <cstdio>
#include <cstdlib>
#include <vector>
#define FQ_S_COUNT_SLOW 1
#include "fq_soft64.h"

long long fq_s_slow_count = 0;
static uint64_t g_s = 99;
static uint64_t rnd()
{
    uint64_t z = (g_s += 0x9e3779b97f4a7c15ULL);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}
static uint64_t few(uint64_t m)
{
    return m & ~((1ULL << (rnd() % 53)) - 1) & 0x000fffffffffffffULL;
}
int main(int argc, char** argv)
{
    const int fam = argc > 1 ? atoi(argv[1]) : 0;
    const long long n = argc > 2 ? atoll(argv[2]) : 100000;
    std::vector<double> f;
    if (fam == 0) {
        f = {0.1, 0.05, 0.005, -0.1, -0.2, 1.0 / 1000, 1.0 / 300007, 1.0, -1.0, 0.25, 3.0, 1.0 / 3.0};
    }
    for (int k = 0; k < 40 && fam > 0; ++k) {
        const uint64_t ends[8] = {0, 1, 2, 1022, 1023, 2045, 2046, 2047};
        uint64_t b = rnd();
        if (fam == 2) {
            b = (b & 0xfff0000000000000ULL) | few(b);
        }
        if (fam == 3) {
            b = (b & 0x8000000000000000ULL) | (ends[rnd() % 8] << 52) | (rnd() & 1 ? 0 : rnd() & 0xfffffffffffffULL);
        }
        f.push_back(fq_from_bits(b));
    }
    long long ops = 0, bad = 0;
    for (double c : f) {
        const fq_sfactor p = fq_s_factor(c);
        for (long long i = 0; i < n; ++i) {
            uint64_t b = rnd();
            if (i & 1) { // around the exponent of 1, few-bit half of the time
                b = (b & 0x800fffffffffffffULL) | ((1023 - 40 + rnd() % 80) << 52);
                b = (i & 2) ? b : (b & 0xfff0000000000000ULL) | few(b);
            }
            const double x = fq_from_bits(b), r = fq_smulc(x, p), w = x * c;
            ++ops;
            bad += !((r != r && w != w) || fq_bits(r) == fq_bits(w));
        }
    }
    printf("%lld %lld %lld\n", ops, bad, fq_s_slow_count);
    return bad ? 1 : 0;
}
