// CPU check of the FP64 butterfly schedule with unsigned twiddles (FpAr in
// csrc/ntt.cuh, the reference's tables): rounds of K <= 4 radix-2 stages from
// normalised values, every product by M2, normalisations where the kernels have
// them (fpar_ct_norm, fpar_gs_norm in csrc/fp_sched.hpp).
// Every operation is the kernel's IEEE double operation (fma correctly
// rounded, no contraction), so the check is bit-exact to the device. Asserted:
// multiplier inputs at most 4q, values below 4.5q + 1 (forward, multiplier inputs
// 2.5q + 1) or 3q + 2 (inverse), every value below 2^53, results normalised, and
// every output equal to 128-bit modular arithmetic, on random inputs and on
// adversarial ones (values at +-q/2, twiddles at 0 and q - 1).
// Usage: fp64_unsigned_rounds <trials per modulus>; exit 0 when clean.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "fp_sched.hpp"

typedef unsigned __int128 u128;
static const double TWO53 = 9007199254740992.0;
static double q, qinv;
static uint64_t Q;
static long violations, mismatches;
static double max_val;

static void bound(double v, double lim) {
    const double a = std::fabs(v);
    if (a > max_val) max_val = a;
    if (a > lim || a >= TWO53) violations++;
}
static double norm(double z) {
    bound(z, TWO53);
    const double k = std::fma(z, qinv, ntt::FP_M1) - ntt::FP_M1;
    return std::fma(-k, q, z);
}
static double mulq(double y, double w) {
    const double h = y * w, l = std::fma(y, w, -h), k = std::fma(h, qinv, ntt::FP_M2) - ntt::FP_M2;
    return std::fma(-k, q, h) + l;
}
static uint64_t rnd64() { return ((uint64_t)rand() << 42) ^ ((uint64_t)rand() << 21) ^ (uint64_t)rand(); }
static uint64_t mm(uint64_t a, uint64_t b) { return (uint64_t)(((u128)a * b) % Q); }
static uint64_t canon(double z) { return (uint64_t)(z < 0.0 ? z + q : z); }

static void round_check(int K, bool inverse, int adv) {
    const int n = 1 << K;
    uint64_t e[16], w[16];
    double v[16];
    for (int u = 0; u < n; ++u) {
        uint64_t x = (adv & 1) ? (Q / 2 + (uint64_t)(rand() % 3)) % Q : rnd64() % Q;
        if ((adv & 1) && (rand() & 1)) x = Q - x;
        v[u] = norm((double)x);
        bound(v[u], 0.5 * q + 1.5);
        e[u] = x;
        w[u] = (adv & 2) ? ((rand() & 1) ? (uint64_t)(rand() % 4) : Q - 1 - (uint64_t)(rand() % 4)) : rnd64() % Q;
    }
    for (int st = 0; st < K; ++st) {
        const int L = inverse ? K - 1 - st : st, half = 1 << (K - 1 - L);
        const double lim = inverse ? 3.0 * q + 2.0 : 4.5 * q + 1.0;
        for (int g = 0; g < (1 << L); ++g) {
            const uint64_t wi = w[((1 << L) + g) & (n - 1)];
            for (int o = 0; o < half; ++o) {
                const int a = g * 2 * half + o, b = a + half;
                const double xx = v[a], yy = v[b];
                const uint64_t ea = e[a], eb = e[b];
                if (!inverse) {
                    bound(yy, 2.5 * q + 1.0);
                    const double r = mulq(yy, (double)wi);
                    v[a] = xx + r;
                    v[b] = xx - r;
                    e[a] = (ea + mm(eb, wi)) % Q;
                    e[b] = (ea + Q - mm(eb, wi)) % Q;
                } else {
                    bound(xx - yy, lim);
                    v[a] = xx + yy;
                    v[b] = mulq(xx - yy, (double)wi);
                    e[a] = (ea + eb) % Q;
                    e[b] = mm((ea + Q - eb) % Q, wi);
                }
                bound(v[a], lim);
                bound(v[b], lim);
            }
        }
        if (inverse ? ntt::fpar_gs_norm(K, L) : ntt::fpar_ct_norm(K, L))
            for (int u = 0; u < n; ++u) v[u] = norm(v[u]);
    }
    for (int u = 0; u < n; ++u) {
        bound(v[u], 0.5 * q + 1.5);
        if (canon(v[u]) != e[u]) mismatches++;
    }
}

int main(int argc, char** argv) {
    // the largest primes below 2^50 that are 1 mod 2^10 (n = 2^9, the worst
    // case of the bounds) and 1 mod 2^17 (n = 2^16), the first 1 mod 2^17
    // prime above 2^49, and a 30-bit NTT prime
    const uint64_t mods[] = {1125899906826241ull, 1125899903827969ull, 562949955125249ull, 1073872897ull};
    const long trials = argc > 1 ? atol(argv[1]) : 100000;
    srand(12345);
    for (int m = 0; m < 4; ++m) {
        Q = mods[m];
        q = (double)Q;
        qinv = 1.0 / q;
        max_val = 0;
        for (long t = 0; t < trials; ++t)
            for (int K = 1; K <= 4; ++K) {
                round_check(K, false, (int)(t & 3));
                round_check(K, true, (int)(t & 3));
            }
        printf("q=%llu: max |value| / q = %.4f\n", (unsigned long long)Q, max_val / q);
    }
    printf("violations=%ld mismatches=%ld\n", violations, mismatches);
    return (violations || mismatches) ? 1 : 0;
}
