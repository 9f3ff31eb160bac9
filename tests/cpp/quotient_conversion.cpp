// CPU check of the FP64-quotient basis conversion with the functions of
// csrc/conv_quot.hpp that the kernels compile in: sum_t x_t c_t mod q for q <
// 2^50 from n sources below 2^b, for every (n, b) that conv_wrap_ok admits.
// Asserted: the first remainder stays inside the signed 64-bit range (recomputed
// in 128 bits), the result is congruent to the 128-bit sum, and |r| <= (1/2 +
// 2^-39) q, inside the normalised bound that the transform takes. Random sources
// and constants, the extremes (sources at 2^b - 1, constants at +-q/2), and
// first remainders beside every half multiple of q that the second step has to
// round. Also the admitted widths themselves.
// Usage: quotient_conversion <trials>; prints violations and mismatches.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include <utility>

#include "conv_quot.hpp"

typedef uint64_t u64;
typedef __int128 i128;

static u64 rnd64() { return ((u64)rand() << 42) ^ ((u64)rand() << 21) ^ (u64)rand(); }

int main(int argc, char** argv) {
    const long trials = argc > 1 ? atol(argv[1]) : 2000;
    const u64 mods[] = {1125899906826241ull, 1125899903827969ull, 562949955125249ull, 1073872897ull};
    long violations = 0, mismatches = 0, forms = 0;
    double worst = 0, far = 0;
    srand(99);
    auto result = [&](i128 sum, int64_t r, u64 q) {
        const double off = std::fabs((double)r) - 0.5 * (double)q;
        if (off > 0x1p-39 * (double)q || std::fabs((double)r) > ntt::B_NORM / 1024.0 * (double)q) violations++;
        if (off > far) far = off;
        if ((sum - (i128)r) % (i128)q != 0) mismatches++;
    };
    for (u64 q : mods) {
        const double qinv = 1.0 / (double)q;
        const pl::WrapConv wc{q, qinv};
        for (int b : {31, 50, 55, 60, 61})
            for (unsigned n = 1; n <= 17; ++n) {
                if (!gfx::conv_wrap_ok(n, 1ull << b)) continue;
                ++forms;
                for (long t = 0; t < trials; ++t) {
                    u64 lo = 0;
                    double s = 0;
                    i128 sum = 0;
                    for (unsigned j = 0; j < n; ++j) {
                        const u64 x = t & 1 ? (1ull << b) - 1 - (u64)(rand() % 3) : rnd64() & ((1ull << b) - 1);
                        const u64 c = t & 2 ? (t & 4 ? q / 2 : q / 2 + 1) : rnd64() % q;
                        const pl::ConvTerm term = j & 1 ? pl::conv_term<true>(c, q, qinv) : pl::conv_term<false>(c, q, qinv);
                        pl::quot_term(lo, s, x, term);
                        const i128 v = (int64_t)term.c;   // +-c, up to a multiple of q
                        if ((v - (j & 1 ? -(i128)c : (i128)c)) % (i128)q != 0) mismatches++;
                        sum += v * (i128)x;
                    }
                    const int64_t k = (int64_t)(pl::q_bits(s + 0x1.8p64) - 0x43F8000000000000ll);
                    const i128 wide = sum - (i128)k * ((i128)q << 12);
                    if (wide != (i128)(int64_t)wide) violations++;
                    const double w = std::fabs((double)wide) / 0x1p63;
                    if (w > worst) worst = w;
                    result(sum, wc.finish(lo, s), q);
                    const double d = wc.finish_d(lo, s);
                    if (d != (double)wc.finish(lo, s)) mismatches++;
                }
            }
        // s = 0: the first remainder is lo itself, taken beside (m + 1/2) q
        for (int m = -7999; m < 7999; ++m)
            for (int d = -300; d <= 300; d += 7) {
                const int64_t r1 = (int64_t)m * (int64_t)q + (int64_t)(q / 2) + d;
                result(r1, wc.finish((u64)r1, 0.0), q);
            }
    }
    for (auto [b, most] : {std::pair<int, unsigned>{60, 10}, {61, 7}}) {
        unsigned n = 0;
        while (gfx::conv_wrap_ok(n + 1, 1ull << b)) ++n;
        if (n != most) { printf("%d bits: %u sources admitted, not %u\n", b, n, most); violations++; }
    }
    if (gfx::conv_wrap_ok(1, 1ull << 62)) violations++;
    printf("forms=%ld largest first remainder %.3f of the 64-bit range, |r| up to q/2 + %.0f\n", forms, worst, far);
    printf("violations=%ld mismatches=%ld\n", violations, mismatches);
    return violations || mismatches ? 1 : 0;
}
