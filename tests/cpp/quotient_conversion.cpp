// CPU check of the FP64-quotient basis conversion (WrapConv in
// csrc/pipeline.cuh) with the kernel's IEEE double operations and 64-bit
// wrap-around products: sum_t x_t c_t mod q for q < 2^50 from n sources below
// 2^b, for every (n, b) that conv_wrap_ok admits. Asserted: the first
// remainder stays inside the signed 64-bit range (recomputed in 128 bits), the
// result is congruent to the 128-bit sum, and |r| <= q/2 + 1. Random sources
// and constants, and the extremes: sources at 2^b - 1, constants at +-q/2.
// Usage: quotient_conversion <trials>; prints violations and mismatches.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>

typedef uint64_t u64;
typedef __int128 i128;

// the rule of csrc/context.hpp
static bool conv_wrap_ok(unsigned n, int b) {
    double unit = std::ldexp(1.0, b - 54);
    return b <= 61 && unit * (0.5 * n * (n + 1) + 2.5 * n) + 2048.0 + 64.0 < 8000.0;
}
static double hl(uint32_t hi, uint32_t lo) {
    const u64 v = (u64)hi << 32 | lo;
    double d;
    std::memcpy(&d, &v, 8);
    return d;
}
static u64 bits(double d) {
    u64 v;
    std::memcpy(&v, &d, 8);
    return v;
}
static double x2d(u64 x) { return (hl(0x45300000, (uint32_t)(x >> 32)) - 0x1.00000001p84) + hl(0x43300000, (uint32_t)x); }
static u64 rnd64() { return ((u64)rand() << 42) ^ ((u64)rand() << 21) ^ (u64)rand(); }

int main(int argc, char** argv) {
    const long trials = argc > 1 ? atol(argv[1]) : 2000;
    const u64 mods[] = {1125899906826241ull, 1125899903827969ull, 562949955125249ull, 1073872897ull};
    const double bias = 0x1p84 + 0x1p63 + 0x1p52, M1 = 6755399441055744.0;
    long violations = 0, mismatches = 0, forms = 0;
    double worst = 0;
    srand(99);
    for (u64 q : mods)
        for (int b : {31, 50, 55, 60, 61})
            for (unsigned n = 1; n <= 17; ++n) {
                if (!conv_wrap_ok(n, b)) continue;
                ++forms;
                const double qinv = 1.0 / (double)q;
                for (long t = 0; t < trials; ++t) {
                    u64 lo = 0;
                    double s = 0;
                    i128 sum = 0;
                    for (unsigned j = 0; j < n; ++j) {
                        const u64 x = t & 1 ? (1ull << b) - 1 - (u64)(rand() % 3) : rnd64() & ((1ull << b) - 1);
                        u64 c = t & 2 ? (t & 4 ? q / 2 : q / 2 + 1) : rnd64() % q;
                        const int64_t v = c > q / 2 ? (int64_t)c - (int64_t)q : (int64_t)c;
                        const double f = (double)v * qinv;
                        lo += x * (u64)v;
                        s = std::fma(x2d(x), f, s);
                        sum += (i128)(int64_t)v * (i128)x;
                    }
                    const int64_t k = (int64_t)(bits(s + 0x1.8p64) - 0x43F8000000000000ull);
                    const u64 r1 = lo - (u64)k * (q << 12);
                    const i128 wide = sum - (i128)k * ((i128)q << 12);
                    if (wide != (i128)(int64_t)r1) violations++;
                    const double h = hl(0x45300000, (uint32_t)(r1 >> 32) ^ 0x80000000u);
                    const double r1d = (h - bias) + hl(0x43300000, (uint32_t)r1);
                    const int32_t k2 = (int32_t)bits(std::fma(r1d, qinv, M1));
                    const int64_t r = (int64_t)(r1 - (u64)(int64_t)k2 * q);
                    if (std::fabs((double)r) > 0.5 * (double)q + 1.0) violations++;
                    const double w = std::fabs((double)wide) / 0x1p63;
                    if (w > worst) worst = w;
                    if ((sum - (i128)r) % (i128)q != 0) mismatches++;
                }
            }
    printf("forms=%ld largest first remainder %.3f of the 64-bit range\n", forms, worst);
    printf("violations=%ld mismatches=%ld\n", violations, mismatches);
    return violations || mismatches ? 1 : 0;
}
