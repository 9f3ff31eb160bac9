// Compile-time schedules of the transform rounds in ntt.cuh: for FpArS, which
// products take the even rounding and which values are normalised, from the
// bounds of a round's inputs; for FpAr and IntAr, the stages that reduce. Plain
// C++, so that the CPU checks of the schedules run the same functions.
#pragma once

#ifdef __CUDACC__
#define GFX_HD __host__ __device__
#else
#define GFX_HD
#endif

namespace ntt {

constexpr double FP_M1 = 6755399441055744.0;    // 1.5 * 2^52
constexpr double FP_M2 = 13510798882111488.0;   // 1.5 * 2^53

// Bounds in units of q / 1024.
constexpr int B_NORM = 514;     // a normalised value, |z| <= q/2 + 1
constexpr int B_CANON = 1024;   // a canonical residue [0, q)
constexpr int B_M1 = 4090;      // multiplier inputs of M1 (below 4q)
constexpr int B_LIM = 8184;     // every value (below 8q < 2^53)
constexpr int B_ROUND = 1990;   // what an inverse round leaves un-normalised
GFX_HD constexpr int mul_bound(int b) { return (b <= B_M1 ? 512 : 1024) + b / 8 + 2; }
// Bound after K forward stages from inputs below b.
GFX_HD constexpr int ct_out(int K, int b) {
    for (int l = 0; l < K; ++l) {
        if (b + mul_bound(b) > B_LIM) b = B_NORM;
        b += mul_bound(b);
    }
    return b;
}
// Schedule of an inverse round of K <= 4 stages from inputs below xin: per
// stage (slot bit s) the slots normalised before it and the pairs (by their
// lower slot) whose product takes M2; the slots normalised at the end so that
// all are below B_ROUND; the largest bound left then, and without that.
struct GsSched {
    unsigned pre[4], even[4], end;
    int out, raw;
};
GFX_HD constexpr GsSched gs_sched(int K, int xin) {
    GsSched S{{0, 0, 0, 0}, {0, 0, 0, 0}, 0, 0, 0};
    int b[16] = {};
    for (int u = 0; u < (1 << K); ++u) b[u] = xin;
    for (int s = 0; s < K; ++s)
        for (int x = 0; x < (1 << K); ++x) {
            if (x >> s & 1) continue;
            const int y = x | (1 << s);
            while (b[x] + b[y] > B_LIM) {
                const int m = b[x] >= b[y] ? x : y;
                S.pre[s] |= 1u << m;
                b[m] = B_NORM;
            }
            const int d = b[x] + b[y];
            if (d > B_M1) S.even[s] |= 1u << x;
            b[x] = d;
            b[y] = mul_bound(d);
        }
    for (int u = 0; u < (1 << K); ++u) {
        S.raw = b[u] > S.raw ? b[u] : S.raw;
        if (b[u] > B_ROUND) {
            S.end |= 1u << u;
            b[u] = B_NORM;
        }
        S.out = b[u] > S.out ? b[u] : S.out;
    }
    return S;
}

// FpAr (unsigned twiddles, every product by M2): whether all values are
// normalised after local stage L of a forward / inverse round of K stages.
GFX_HD constexpr bool fpar_ct_norm(int K, int L) { return L % 2 == 1 || L == K - 1; }
GFX_HD constexpr bool fpar_gs_norm(int K, int L) { return (K - L) % 2 == 0 || L == 0; }

// IntAr: whether a forward stage brings its untouched operand below 4q; whether
// the pair at offset o of an inverse stage of half 2^s adds two sums (below 4q,
// reduced) rather than two products (below 2q).
GFX_HD constexpr bool int_ct_reduces(int L) { return L % 2 == 0; }
GFX_HD constexpr bool int_gs_sums(int s, int o) { return s > 0 && (o >> (s > 0 ? s - 1 : 0) & 1) == 0; }

GFX_HD constexpr int cmin(int a, int b) { return a < b ? a : b; }
GFX_HD constexpr int cmax(int a, int b) { return a > b ? a : b; }

// Bounds (FpArS) of a forward column pass's results from inputs below X0, and
// of an inverse row pass's.
template <class AR>
GFX_HD constexpr int fwd_col_bound(int A, int X0) {
    for (int j = 0; j < A; j += 4) X0 = AR::fwd_out(cmin(4, A - j), X0);
    return X0;
}
template <class AR>
GFX_HD constexpr int inv_row_bound(int X0) { return AR::inv_out(4, AR::inv_out(4, X0)); }

}  // namespace ntt

namespace pl {

// Bounds of the pipeline's transform inputs on the FP64 path: P1's tensor
// products of canonical operands stay below 1.25q, P3's converted digits are
// normalised, canonical or a sum of at most three signed products (0.63q each),
// P8's prologue is normalised, U is canonical.
constexpr int P1_IN = 1290, P3_IN = 1930, P8_IN = ntt::B_NORM, P6_IN = ntt::B_CANON;

}  // namespace pl
