// CPU check of the integer butterfly schedule for packed tables (IntAr in
// csrc/ntt.cuh, reductions by int_ct_reduces and int_gs_sums of
// csrc/fp_sched.hpp): rounds of one to four stages, forward from values below 8q,
// inverse from values below 2q, for primes up to just below 2^61. Asserted: no sum
// or difference leaves [0, 8q) or 64 bits (recomputed in 128 bits), forward
// results stay below 8q and inverse ones below 2q, and every result is congruent
// to 128-bit arithmetic. Random inputs and the ends of their range, twiddles at 0,
// 1 and q - 1. Usage: int_round_bounds <trials>; exit 0 when clean.
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "fp_sched.hpp"

typedef uint64_t u64;
typedef unsigned __int128 u128;
static u64 Q;
static long violations, mismatches;

static u64 rnd64() { return ((u64)rand() << 42) ^ ((u64)rand() << 21) ^ (u64)rand(); }
static u64 mm(u64 a, u64 b) { return (u64)((u128)a * b % Q); }
static u64 csub(u64 x, u64 m) { return x >= m ? x - m : x; }
// w x mod q in [0, 2q) for any 64-bit x (Shoup)
static u64 shoup_lazy(u64 x, u64 w) {
    const u64 wp = (u64)(((u128)w << 64) / Q);
    return x * w - (u64)((u128)x * wp >> 64) * Q;
}
static u64 within(u128 v, u128 lim) {   // also catches a negative difference: it wraps far above lim
    if (v >= lim) violations++;
    return (u64)v;
}

static void round_check(int K, bool inverse, int adv) {
    const int n = 1 << K;
    const u128 q = Q;
    u64 v[16], e[16], w[16];
    for (int u = 0; u < n; ++u) {
        const u64 top = inverse ? 2 * Q : 8 * Q;
        v[u] = adv & 1 ? (rand() & 1 ? top - 1 - (u64)(rand() % 2) : (u64)(rand() % 2)) : rnd64() % top;
        e[u] = v[u] % Q;
        const u64 edge[] = {0, 1, Q - 1};
        w[u] = adv & 2 ? edge[rand() % 3] : rnd64() % Q;
    }
    for (int st = 0; st < K; ++st) {
        const int L = inverse ? K - 1 - st : st, s = K - 1 - L, half = 1 << s;
        for (int g = 0; g < (1 << L); ++g)
            for (int o = 0; o < half; ++o) {
                const int a = g * 2 * half + o, b = a + half;
                const u64 t = w[((1 << L) + g) & (n - 1)], ea = e[a], eb = e[b];
                if (!inverse) {
                    const u64 xx = ntt::int_ct_reduces(L) ? csub(v[a], 4 * Q) : v[a];
                    const u64 r = within(shoup_lazy(v[b], t), 2 * q);
                    v[a] = within((u128)xx + r, 8 * q);
                    v[b] = within((u128)xx - r + 2 * q, 8 * q);
                    e[a] = (u64)(((u128)ea + mm(eb, t)) % q);
                    e[b] = (u64)(((u128)ea + q - mm(eb, t)) % q);
                } else {
                    const bool sums = ntt::int_gs_sums(s, o);
                    const u64 d = within((u128)v[a] - v[b] + (sums ? 4 : 2) * q, 8 * q);
                    const u64 x = within((u128)v[a] + v[b], 8 * q);
                    v[a] = within(sums ? csub(x, 4 * Q) : x, 4 * q);
                    v[b] = within(shoup_lazy(d, t), 2 * q);
                    e[a] = (u64)(((u128)ea + eb) % q);
                    e[b] = mm((u64)(((u128)ea + q - eb) % q), t);
                }
            }
    }
    for (int u = 0; u < n; ++u) {
        if (inverse && u < n / 2) v[u] = csub(v[u], 2 * Q);
        within(v[u], inverse ? 2 * q : 8 * q);
        if (v[u] % Q != e[u]) mismatches++;
    }
}

int main(int argc, char** argv) {
    const long trials = argc > 1 ? atol(argv[1]) : 20000;
    // just below 2^61 and 2^60 (the bounds need no NTT prime: any odd modulus), a 50- and a 30-bit prime
    const u64 mods[] = {(1ull << 61) - 1, (1ull << 60) - 93, 1125899906826241ull, 1073872897ull};
    srand(4321);
    for (u64 m : mods) {
        Q = m;
        for (long t = 0; t < trials; ++t)
            for (int K = 1; K <= 4; ++K) {
                round_check(K, false, (int)(t & 3));
                round_check(K, true, (int)(t & 3));
            }
    }
    printf("violations=%ld mismatches=%ld\n", violations, mismatches);
    return violations || mismatches ? 1 : 0;
}
