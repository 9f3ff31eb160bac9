// Host helpers (include/host_ops.h, keygen.h) on moduli up to 2^62, written as
// a caller of the C++ API writes them. For every ring size and for primes just
// below 2^62, 2^61 and 2^50: pt_to_eval_host at sampled slots equals the
// plaintext's value at psi^(2 brv(j) + 1) computed from the definition, and
// decrypt_host with a zero secret returns the plaintext it came from. Messages
// hold both ends of the 64-bit range. Prints one line per ring; exit 0 when
// all agree.
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "host_ops.h"
#include "keygen.h"
#include "params.h"

using u64 = uint64_t;
using u128 = unsigned __int128;

static u64 residue(int64_t v, u64 q) {
    const __int128 r = (__int128)v % (__int128)q;
    return (u64)(r < 0 ? r + (__int128)q : r);
}
static u64 power(u64 b, u64 e, u64 q) {
    u64 r = 1;
    for (; e; e >>= 1, b = (u64)((u128)b * b % q))
        if (e & 1) r = (u64)((u128)r * b % q);
    return r;
}

int main() {
    long bad = 0;
    std::mt19937_64 rng(7);
    for (uint32_t logn = 9; logn <= 16; ++logn) {
        const uint32_t n = 1u << logn;
        std::vector<u64> mod, root;
        for (uint32_t bits : {62u, 61u, 50u}) {
            std::vector<u64> p;
            gpufhe::native_primes(p, 1, bits, n, {});
            mod.push_back(p[0]);
            root.push_back(gpufhe::native_root(n, p[0]));
        }
        std::vector<int64_t> m(n);
        for (auto& v : m) v = (int64_t)rng();
        m[0] = INT64_MAX;
        m[1] = INT64_MIN + 1;
        m[n - 1] = -1;
        std::vector<u64> ev;
        gpufhe::pt_to_eval_host(ev, m, (uint32_t)mod.size(), n, mod, root);
        long fwd = 0, inv = 0;
        for (size_t t = 0; t < mod.size(); ++t) {
            const u64 q = mod[t];
            for (int k = 0; k < 32; ++k) {
                const uint32_t j = k == 0 ? 0 : k == 1 ? n - 1 : (uint32_t)(rng() % n);
                uint32_t br = 0;
                for (uint32_t b = 0; b < logn; ++b) br |= (j >> b & 1) << (logn - 1 - b);
                const u64 x = power(root[t], 2ull * br + 1, q);
                u64 s = 0;
                for (uint32_t i = n; i-- > 0;) s = (u64)(((u128)s * x + residue(m[i], q)) % q);
                fwd += s != ev[t * n + j];
            }
            const std::vector<u64> c0(ev.begin() + t * n, ev.begin() + (t + 1) * n), zero(n, 0);
            std::vector<int64_t> back;
            gpufhe::decrypt_host(back, c0, zero, zero, n, {q}, {root[t]});
            for (uint32_t i = 0; i < n; ++i) inv += residue(back[i], q) != residue(m[i], q);
        }
        std::printf("n=%u forward mismatches=%ld inverse mismatches=%ld\n", n, fwd, inv);
        bad += fwd + inv;
    }
    std::printf("mismatches=%ld\n", bad);
    return bad ? 1 : 0;
}
