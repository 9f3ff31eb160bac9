// CPU check of the bound-scheduled FP64 rounds (FpArS in csrc/ntt.cuh): every
// forward and inverse round of one to four stages, from every input bound that
// occurs in a transform of 2^9 .. 2^16 points, follows the kernel's own
// compile-time schedule (csrc/fp_sched.hpp) with the kernel's IEEE double
// operations. Asserted on random and adversarial values (inputs at the ends of
// their bound, twiddles at +-(q-1)/2): multiplier inputs below 2^52 (M1) or
// 2^53 (M2), every value an integer below 2^53 and within the bound that the
// schedule tracks, and every result equal to 128-bit modular arithmetic.
// Usage: fp64_round_schedule <trials>; prints violations and mismatches.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <set>

#include "fp_sched.hpp"

typedef unsigned __int128 u128;
typedef uint64_t u64;
static const double M1 = ntt::FP_M1, M2 = ntt::FP_M2;
static const double TWO52 = 4503599627370496.0, TWO53 = 9007199254740992.0;
static double q, qinv;
static u64 Q;
static long violations, mismatches;
static double slack = 1e9;

static void below(double v, double lim) {
    if (!(std::fabs(v) < lim)) violations++;
}
static void tracked(double v, int b) {   // within b/1024 q (two units of rounding)
    const double room = b / 1024.0 * q + 2.0 - std::fabs(v);
    if (room < 0) violations++;
    if (room / q < slack) slack = room / q;
}
static double norm(double z) {
    below(z, TWO53);
    const double k = std::fma(z, qinv, M1) - M1;
    return std::fma(-k, q, z);
}
static double mulq(double y, double w, bool even) {
    below(y, even ? TWO53 : TWO52);
    const double M = even ? M2 : M1;
    const double h = y * w, l = std::fma(y, w, -h), k = std::fma(h, qinv, M) - M;
    return std::fma(-k, q, h) + l;
}
static u64 rnd64() { return ((u64)rand() << 42) ^ ((u64)rand() << 21) ^ (u64)rand(); }
static u64 mm(u64 a, u64 b) { return (u64)(((u128)a * b) % Q); }
static u64 res(double z) {   // integer |z| < 2^53 -> [0, q)
    const long long v = (long long)z % (long long)Q;
    return (u64)(v < 0 ? v + (long long)Q : v);
}

static void round_check(int K, bool inverse, int bin, int adv) {
    const int n = 1 << K;
    double v[16], w[16];
    u64 e[16], wi[16];
    int b[16];
    for (int u = 0; u < n; ++u) {
        double z = std::floor(bin / 1024.0 * q * (adv & 1 ? 1.0 : (double)(rnd64() >> 12) * 0x1p-52));
        if (z >= TWO53) z = TWO53 - 1;
        z -= adv & 1 ? (double)(rand() % 3) : 0.0;
        v[u] = rand() & 1 ? -z : z;
        e[u] = res(v[u]);
        b[u] = bin;
        const u64 t = adv & 2 ? Q / 2 + (u64)(rand() & 1) - (u64)(2 * (rand() & 1)) : rnd64() % Q;
        wi[u] = t;
        w[u] = t > Q / 2 ? -(double)(Q - t) : (double)t;
    }
    const ntt::GsSched S = ntt::gs_sched(K, bin);
    for (int st = 0; st < K; ++st) {
        const int L = inverse ? K - 1 - st : st, half = 1 << (K - 1 - L);
        if (!inverse && b[0] + ntt::mul_bound(b[0]) > ntt::B_LIM)
            for (int u = 0; u < n; ++u) { v[u] = norm(v[u]); b[u] = ntt::B_NORM; tracked(v[u], b[u]); }
        const int bs = b[0];
        for (int g = 0; g < (1 << L); ++g)
            for (int o = 0; o < half; ++o) {
                const int x = g * 2 * half + o, y = x + half, t = ((1 << L) + g) & (n - 1);
                const u64 ex = e[x], ey = e[y];
                if (!inverse) {
                    const double r = mulq(v[y], w[t], bs > ntt::B_M1), xx = v[x];
                    v[x] = xx + r;
                    v[y] = xx - r;
                    b[x] = b[y] = bs + ntt::mul_bound(bs);
                    e[x] = (ex + mm(ey, wi[t])) % Q;
                    e[y] = (ex + Q - mm(ey, wi[t])) % Q;
                } else {
                    if (S.pre[st] >> x & 1) { v[x] = norm(v[x]); b[x] = ntt::B_NORM; }
                    if (S.pre[st] >> y & 1) { v[y] = norm(v[y]); b[y] = ntt::B_NORM; }
                    const double xx = v[x], yy = v[y];
                    below(xx - yy, TWO53);
                    v[x] = xx + yy;
                    v[y] = mulq(xx - yy, w[t], S.even[st] >> x & 1);
                    const int d = b[x] + b[y];
                    b[x] = d;
                    b[y] = ntt::mul_bound(d);
                    e[x] = (ex + ey) % Q;
                    e[y] = mm((ex + Q - ey) % Q, wi[t]);
                }
                below(v[x], TWO53);
                below(v[y], TWO53);
                tracked(v[x], b[x]);
                tracked(v[y], b[y]);
                if (b[x] > ntt::B_LIM || b[y] > ntt::B_LIM) violations++;
            }
    }
    for (int u = 0; u < n; ++u) {
        if (inverse && b[u] > S.raw) violations++;
        if (inverse && (S.end >> u & 1)) { v[u] = norm(v[u]); b[u] = ntt::B_NORM; tracked(v[u], b[u]); }
        if (inverse && b[u] > S.out) violations++;
        if (!inverse && b[u] != ntt::ct_out(K, bin)) violations++;
        if (res(v[u]) != e[u]) mismatches++;
    }
}

struct Fwd { static constexpr int fwd_out(int K, int b) { return ntt::ct_out(K, b); } };

int main(int argc, char** argv) {
    const u64 mods[] = {1125899906826241ull, 1125899903827969ull, 562949955125249ull, 1073872897ull};
    const long trials = argc > 1 ? atol(argv[1]) : 2000;
    // input bounds of the kernels: normalised, canonical, tensor products, sums of three converted products
    const int starts[] = {pl::P8_IN, pl::P6_IN, pl::P1_IN, pl::P3_IN};
    std::set<int> fwd[5], inv[5];
    for (int x0 : starts)
        for (int A = 1; A <= 8; ++A) {
            int b = x0;
            for (int j = 0; j < A; j += 4) { const int K = ntt::cmin(4, A - j); fwd[K].insert(b); b = ntt::ct_out(K, b); }
            if (b != ntt::fwd_col_bound<Fwd>(A, x0)) violations++;
            fwd[4].insert(b);
            fwd[4].insert(ntt::ct_out(4, b));
            b = x0;
            for (int i = 0; i < 2; ++i) { inv[4].insert(b); b = ntt::gs_sched(4, b).out; }
            for (int JE = A; JE > 0; JE = ((JE - 1) / 4) * 4) {
                const int K = JE - ((JE - 1) / 4) * 4;
                inv[K].insert(b);
                b = ntt::gs_sched(K, b).out;
            }
        }
    srand(12345);
    for (u64 m : mods) {
        Q = m;
        q = (double)Q;
        qinv = 1.0 / q;
        for (int K = 1; K <= 4; ++K)
            for (long t = 0; t < trials; ++t) {
                for (int b : fwd[K]) round_check(K, false, b, (int)(t & 3));
                for (int b : inv[K]) round_check(K, true, b, (int)(t & 3));
            }
    }
    printf("least room below a tracked bound: %.4f q\n", slack);
    printf("violations=%ld mismatches=%ld\n", violations, mismatches);
    return violations || mismatches ? 1 : 0;
}
