// Compile-time schedule of the FP64 transform rounds (FpArS in ntt.cuh): which
// products take the even rounding and which values are normalised, from the
// bounds of a round's inputs. Plain C++, so that the CPU check of the schedule
// runs the same functions.
#pragma once

#ifdef __CUDACC__
#define GFX_HD __host__ __device__
#else
#define GFX_HD
#endif

namespace ntt {

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
