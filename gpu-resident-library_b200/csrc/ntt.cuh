// Two-pass negacyclic NTT engine for N = 2^LOGN, 9 <= LOGN <= 16.
//
// The transform is the reference's: forward Cooley-Tukey with twiddle
// roots[m+i] = psi^bitrev(m+i) (standard order in, bit-reversed out) and the
// inverse Gentleman-Sande with the same indexing (bit-reversed in, standard
// out). The coefficient vector is viewed as a matrix x[r*256 + c] with
// R1 = 2^(LOGN-8) rows of 256 columns:
//   * the first A = LOGN-8 forward stages only couple rows (fixed column):
//     the "column pass", tile = all R1 rows x C columns;
//   * the last 8 stages only couple columns inside one row: the "row pass",
//     tile = RB rows x 256.
// Each pass runs radix-2^K rounds held in registers (K <= 4, 16 values per
// thread), exchanging through shared memory between rounds, so a pass reads
// and writes global memory once.
//
// Two arithmetic policies run the same rounds. IntAr: 64-bit integer
// Harvey lazy butterflies with Shoup twiddles (forward values in [0,8q),
// inverse in [0,2q)), q < 2^61 (IntArWide: [0,4q), q < 2^62). FpArS and FpAr
// (q < 2^50): residues held as signed FP64 integers and multiplied exactly with
// FMA, which runs on the FP64 pipe at about twice the integer path's butterfly
// rate. Both give the same canonical residues, so callers pick per tower.
//
// Twiddle index of line-local stage j: a round that starts at stage J0 with
// group base B = 2^(goff+J0) + HB uses twiddle (B << l) + (u >> (K-l)) at its
// local stage l for register slot u (see ct_reg / gs_reg).
#pragma once
#include "fp_sched.hpp"
#include "gf.cuh"

namespace ntt {

struct TwPacked {
    const Tw* t;
    __device__ __forceinline__ Tw operator()(u32 i) const { return t[i]; }
};
struct TwSplit {
    const u64* w;
    const u64* wp;
    __device__ __forceinline__ Tw operator()(u32 i) const { return Tw{__ldg(w + i), __ldg(wp + i)}; }
};

// FP64 twiddle accessors: a library double table, or the reference's u64
// table converted on load.
__device__ __forceinline__ double u2d(u64 x) {   // exact for x < 2^52
    return __dsub_rn(__longlong_as_double((long long)(x | 0x4330000000000000ull)), 4503599627370496.0);
}
__device__ __forceinline__ u64 d2u(double z) {   // integer 0 <= z < 2^52
    return (u64)__double_as_longlong(__dadd_rn(z, 4503599627370496.0)) & 0xFFFFFFFFFFFFFull;
}
struct TwD {
    const double* t;
    __device__ __forceinline__ double operator()(u32 i) const { return __ldg(t + i); }
};

// The 2^L twiddles tw(base + g), g < 2^L, of one butterfly group at local
// stage L (base = B << L, so the run is aligned to 2^L entries). The
// library's double tables (TwD, 16-byte aligned per modulus) load them as
// 16-byte vectors; other tables load word by word.
template <int L, class TW>
__device__ __forceinline__ void tw_run(const TW& tw, u32 base, double (&w)[1 << L]) {
#pragma unroll
    for (int g = 0; g < (1 << L); ++g) w[g] = tw(base + (u32)g);
}
template <int L>
__device__ __forceinline__ void tw_run(const TwD& tw, u32 base, double (&w)[1 << L]) {
    if constexpr (L == 0) {
        w[0] = __ldg(tw.t + base);
    } else {
        const double2* p = reinterpret_cast<const double2*>(tw.t + base);
#pragma unroll
        for (int h = 0; h < (1 << (L - 1)); ++h) {
            const double2 v = __ldg(p + h);
            w[2 * h] = v.x;
            w[2 * h + 1] = v.y;
        }
    }
}
struct TwDConv {
    const u64* w;
    __device__ __forceinline__ double operator()(u32 i) const { return u2d(__ldg(w + i)); }
};

// One radix-2 stage (local stage L of K) on the register slots; recursion
// over L keeps every index a compile-time constant so v stays in registers.
template <int K, int L, class TW>
__device__ __forceinline__ void ct_stage(u64 (&v)[1 << K], const TW& tw, u32 B, u64 q, u64 two_q) {
    constexpr int half = 1 << (K - 1 - L);
#pragma unroll
    for (int g = 0; g < (1 << L); ++g) {
        const Tw t = tw((B << L) + g);
#pragma unroll
        for (int o = 0; o < half; ++o)
            ct_bfly(v[g * 2 * half + o], v[g * 2 * half + o + half], t.w, t.wp, q, two_q);
    }
    if constexpr (L + 1 < K) ct_stage<K, L + 1>(v, tw, B, q, two_q);
}

template <int K, int L, class TW>
__device__ __forceinline__ void gs_stage(u64 (&v)[1 << K], const TW& tw, u32 B, u64 q, u64 two_q) {
    constexpr int half = 1 << (K - 1 - L);
#pragma unroll
    for (int g = 0; g < (1 << L); ++g) {
        const Tw t = tw((B << L) + g);
#pragma unroll
        for (int o = 0; o < half; ++o)
            gs_bfly(v[g * 2 * half + o], v[g * 2 * half + o + half], t.w, t.wp, q, two_q);
    }
    if constexpr (L > 0) gs_stage<K, L - 1>(v, tw, B, q, two_q);
}

// K forward stages (local 0..K-1) / K inverse stages (local K-1..0).
template <int K, class TW>
__device__ __forceinline__ void ct_reg(u64 (&v)[1 << K], const TW& tw, u32 B, u64 q, u64 two_q) {
    ct_stage<K, 0>(v, tw, B, q, two_q);
}
template <int K, class TW>
__device__ __forceinline__ void gs_reg(u64 (&v)[1 << K], const TW& tw, u32 B, u64 q, u64 two_q) {
    gs_stage<K, K - 1>(v, tw, B, q, two_q);
}

// ------------------------------------------------------------------ FP64 arithmetic
// Residues as FP64 integers for q < 2^50 (so 8q < 2^53). With
// M2 = 1.5*2^53 and M1 = 1.5*2^52 ("magic" constants whose addition rounds
// to the nearest even / nearest integer) and qinv = RN(1/q) (relative error
// at most 2^-53):
//   mul(y, w): h = RN(y*w); l = y*w - h exactly (FMA); k = RN(h*qinv) by M1
//     or RN2(h*qinv) (even) by M2; r = (h - k*q) + l. h, l, h - k*q and r are
//     exact integers (|h| >= 2^53 makes h an integer, h - k*q and r are
//     integers below 2^52), so r = y*w (mod q). With |h| <= c*q*|w|:
//     |l| <= |h| 2^-53 and |k - h/q| <= e + |h/q| 2^-53, e = 1/2 (M1) or 1 (M2).
//   norm(z), |z| < 2^53: k = RN(z*qinv) by M1; z - k*q in [-q/2 - 1, q/2 + 1].
//
// Unsigned twiddles 0 <= w < q (FpAr, tables converted on load): mul
// by M2 for |y| <= 4q gives |r| <= 2q. A round keeps every value normalised
// at its start and end and normalises after every second stage: forward (CT)
// values stay below 4.5q + 1 and multiplier inputs below 2.5q + 1; inverse
// (GS) values below 3q + 2, multiplier inputs below 3q + 2.
//
// Signed twiddles |w| <= (q-1)/2 (FpArS, the library's double tables): |h/q|
// <= |y|/2, so with c = |y|/q and q < 2^50, |l| <= (c/16) q and
//   M1 (needs |y| < 2^52, c <= 4):  |r| <= (1/2 + c/8) q,
//   M2 (needs |y| < 2^53, c <= 8):  |r| <= (1 + c/8) q.
// A value therefore stays exact while it is below 8q, whatever its round, and
// a multiplied value falls back to 2q or less by itself. So the stages are
// scheduled at compile time from the bound of their inputs (mul_bound,
// ct_out, gs_sched; in units of q / 1024): each stage takes M1 while its
// multiplier inputs are below 4q, else M2, and a value is normalised (three
// operations) only before a sum that could reach 8q, and where a transform
// ends. Forward (CT): 1.0q -> 1.63, 2.34, 3.13, 4.02, 5.53, 7.2q over six
// stages, so 16 stages normalise each value three times, the last of them for
// the output, where one normalisation per round of four and one on load are
// five. Inverse (GS): sums double, products do not, so each radix slot has a
// bound of its own and a round of four normalises 4 slots before its third
// stage and 8 at its end instead of 16. Every value stays an exact integer
// below 2^53, so the results equal the integer path's canonical residues.
// The FP64 pipe is what these passes load most (54-71% busy). Measured with
// this schedule, the scale of the inverse taken on the un-normalised value and
// the row walks below, before -> after: 64 x 12 towers of 2^16, products and
// inverse 650 -> 622 us, embedding 425 -> 415 us; phases of 128 products P1 355
// -> 336, P2 270 -> 247, P3 1510 -> 1456, P4 1036 -> 1012 us.
struct FpBase {
    using T = double;
    double q, qinv;
    u64 qi;                      // q as an integer
    __device__ __forceinline__ double norm(double z) const {
        const double k = __dsub_rn(__fma_rn(z, qinv, FP_M1), FP_M1);
        return __fma_rn(-k, q, z);
    }
    template <bool EVEN = true>
    __device__ __forceinline__ double mulq(double y, double w) const {
        constexpr double M = EVEN ? FP_M2 : FP_M1;
        const double h = __dmul_rn(y, w);
        const double l = __fma_rn(y, w, -h);
        const double k = __dsub_rn(__fma_rn(h, qinv, M), M);
        return __dadd_rn(__fma_rn(-k, q, h), l);
    }
    // x < 4q (any lazy residue of the integer kernels) -> normalised
    __device__ __forceinline__ double in(u64 x) const { return norm(u2d(x)); }
    __device__ __forceinline__ double in_canon(u64 x) const { return u2d(x); }   // x in [0, q)
    // normalised z -> canonical [0, q): one FP64 addition puts z, biased, into
    // the low mantissa bits; the sign is fixed on the integer pipes
    __device__ __forceinline__ u64 out(double z) const {
        const long long v = __double_as_longlong(__dadd_rn(z, FP_M1)) - 0x4338000000000000ll;
        return (u64)(v < 0 ? v + (long long)qi : v);
    }
    __device__ __forceinline__ u64 bits(double z) const { return (u64)__double_as_longlong(z); }
    __device__ __forceinline__ double unbits(u64 b) const { return __longlong_as_double((long long)b); }
    // residue [0, q) -> signed double in (-q/2, q/2]
    __device__ __forceinline__ double sgn(u64 x) const {
        return u2d(x) - (x > (qi >> 1) ? q : 0.0);
    }
    // final word of a forward transform (normalised) -> canonical, also where [0, 2q) would do
    __device__ __forceinline__ u64 final_canon(u64 b) const { return out(unbits(b)); }
    __device__ __forceinline__ u64 final_2q(u64 b) const { return out(unbits(b)); }
    // any |z| < 8q -> canonical
    __device__ __forceinline__ u64 canon(double z) const { return out(norm(z)); }
};

// Unsigned twiddles (the reference's u64 tables converted on load): every
// round starts and ends normalised (see above); its bounds do not travel.
struct FpAr : FpBase {
    __host__ __device__ static constexpr int fwd_out(int, int) { return 0; }
    __host__ __device__ static constexpr int inv_out(int, int) { return 0; }
    __device__ __forceinline__ FpAr(double q_, double qinv_, u64 qi_) : FpBase{q_, qinv_, qi_} {}
    template <int K, int L, class TW>
    __device__ __forceinline__ void ct_stage(double (&v)[1 << K], const TW& tw, u32 B) const {
        static_assert(K <= 4, "bounds are proven for rounds of at most four stages");
        constexpr int half = 1 << (K - 1 - L);
        double wr[1 << L];
        tw_run<L>(tw, B << L, wr);
#pragma unroll
        for (int g = 0; g < (1 << L); ++g) {
            const double w = wr[g];
#pragma unroll
            for (int o = 0; o < half; ++o) {
                double& x = v[g * 2 * half + o];
                double& y = v[g * 2 * half + o + half];
                const double r = mulq<true>(y, w), xx = x;
                x = __dadd_rn(xx, r);
                y = __dsub_rn(xx, r);
            }
        }
        if constexpr (fpar_ct_norm(K, L)) {
#pragma unroll
            for (int u = 0; u < (1 << K); ++u) v[u] = norm(v[u]);
        }
        if constexpr (L + 1 < K) ct_stage<K, L + 1>(v, tw, B);
    }
    template <int K, int L, class TW>
    __device__ __forceinline__ void gs_stage(double (&v)[1 << K], const TW& tw, u32 B) const {
        static_assert(K <= 4, "bounds are proven for rounds of at most four stages");
        constexpr int half = 1 << (K - 1 - L);
        double wr[1 << L];
        tw_run<L>(tw, B << L, wr);
#pragma unroll
        for (int g = 0; g < (1 << L); ++g) {
            const double w = wr[g];
#pragma unroll
            for (int o = 0; o < half; ++o) {
                double& x = v[g * 2 * half + o];
                double& y = v[g * 2 * half + o + half];
                const double xx = x, yy = y;
                x = __dadd_rn(xx, yy);
                y = mulq<true>(__dsub_rn(xx, yy), w);
            }
        }
        if constexpr (fpar_gs_norm(K, L)) {
#pragma unroll
            for (int u = 0; u < (1 << K); ++u) v[u] = norm(v[u]);
        }
        if constexpr (L > 0) gs_stage<K, L - 1>(v, tw, B);
    }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void fwd(double (&v)[1 << K], const TW& tw, u32 B) const { ct_stage<K, 0>(v, tw, B); }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void inv(double (&v)[1 << K], const TW& tw, u32 B) const { gs_stage<K, K - 1>(v, tw, B); }
};

// Signed twiddles in (-q/2, q/2) (the library's double tables), scheduled by
// bounds: BIN = bound of the inputs; END = this round's results are the
// forward transform's (normalised) / need no bound for a next round (inverse).
struct FpArS : FpBase {
    __host__ __device__ static constexpr int fwd_out(int K, int b) { return ct_out(K, b); }
    __host__ __device__ static constexpr int inv_out(int K, int b) { return gs_sched(K, b).out; }
    __device__ __forceinline__ FpArS(double q_, double qinv_, u64 qi_) : FpBase{q_, qinv_, qi_} {}
    template <int K, int L, int BIN, bool END, class TW>
    __device__ __forceinline__ void ct_stage(double (&v)[1 << K], const TW& tw, u32 B) const {
        constexpr int half = 1 << (K - 1 - L);
        constexpr bool PRE = BIN + mul_bound(BIN) > B_LIM;
        constexpr int b = PRE ? B_NORM : BIN;
        static_assert(b + mul_bound(b) <= B_LIM, "forward bound");
        constexpr bool EVEN = b > B_M1;
        if constexpr (PRE) {
#pragma unroll
            for (int u = 0; u < (1 << K); ++u) v[u] = norm(v[u]);
        }
        double wr[1 << L];
        tw_run<L>(tw, B << L, wr);
#pragma unroll
        for (int g = 0; g < (1 << L); ++g) {
            const double w = wr[g];
#pragma unroll
            for (int o = 0; o < half; ++o) {
                double& x = v[g * 2 * half + o];
                double& y = v[g * 2 * half + o + half];
                const double r = mulq<EVEN>(y, w), xx = x;
                x = __dadd_rn(xx, r);
                y = __dsub_rn(xx, r);
            }
        }
        if constexpr (L + 1 < K) {
            ct_stage<K, L + 1, b + mul_bound(b), END>(v, tw, B);
        } else if constexpr (END) {
#pragma unroll
            for (int u = 0; u < (1 << K); ++u) v[u] = norm(v[u]);
        }
    }
    template <int K, int L, int BIN, bool END, class TW>
    __device__ __forceinline__ void gs_stage(double (&v)[1 << K], const TW& tw, u32 B) const {
        constexpr int s = K - 1 - L, half = 1 << s;
        constexpr unsigned pre = gs_sched(K, BIN).pre[s], even = gs_sched(K, BIN).even[s], end = gs_sched(K, BIN).end;
        double wr[1 << L];
        tw_run<L>(tw, B << L, wr);
#pragma unroll
        for (int g = 0; g < (1 << L); ++g) {
            const double w = wr[g];
#pragma unroll
            for (int o = 0; o < half; ++o) {
                const int i = g * 2 * half + o;
                double& x = v[i];
                double& y = v[i + half];
                if (pre >> i & 1) x = norm(x);
                if (pre >> (i + half) & 1) y = norm(y);
                const double xx = x, yy = y, d = __dsub_rn(xx, yy);
                x = __dadd_rn(xx, yy);
                y = (even >> i & 1) ? mulq<true>(d, w) : mulq<false>(d, w);
            }
        }
        if constexpr (L > 0) {
            gs_stage<K, L - 1, BIN, END>(v, tw, B);
        } else if constexpr (!END) {
#pragma unroll
            for (int u = 0; u < (1 << K); ++u)
                if (end >> u & 1) v[u] = norm(v[u]);
        }
    }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void fwd(double (&v)[1 << K], const TW& tw, u32 B) const {
        ct_stage<K, 0, BIN, END>(v, tw, B);
    }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void inv(double (&v)[1 << K], const TW& tw, u32 B) const {
        gs_stage<K, K - 1, BIN, END>(v, tw, B);
    }
};

// Integer path for any q < 2^62 (the reference's tables): the lazy Harvey/Shoup
// butterflies above, values as-is.
struct IntArWide {
    using T = u64;
    u64 q, two_q;
    __host__ __device__ static constexpr int fwd_out(int, int) { return 0; }
    __host__ __device__ static constexpr int inv_out(int, int) { return 0; }
    __device__ __forceinline__ u64 in(u64 x) const { return x; }
    __device__ __forceinline__ u64 in_canon(u64 x) const { return x; }
    __device__ __forceinline__ u64 bits(u64 x) const { return x; }
    __device__ __forceinline__ u64 unbits(u64 b) const { return b; }
    // lazy [0, 4q) -> canonical [0, q), or -> [0, 2q)
    __device__ __forceinline__ u64 final_canon(u64 b) const { return csub(csub(b, two_q), q); }
    __device__ __forceinline__ u64 final_2q(u64 b) const { return csub(b, two_q); }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void fwd(u64 (&v)[1 << K], const TW& tw, u32 B) const { ct_reg<K>(v, tw, B, q, two_q); }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void inv(u64 (&v)[1 << K], const TW& tw, u32 B) const { gs_reg<K>(v, tw, B, q, two_q); }
};

// Integer path of the library's tables, q < 2^61, so 8q fits 64 bits. Forward
// values stay below 8q: a Shoup product is below 2q for any 64-bit operand, so
// only the untouched operand needs reducing, and every second stage is enough
// (4q -> 6q -> 8q). Inverse values enter and leave a round below 2q: a sum is
// reduced only where both its operands are sums (csub where they are below 4q),
// by radix slot, 20 conditional subtractions per round of four instead of 32.
// A 64-bit conditional subtraction is ten issue cycles of the butterfly's fifty
// (measured); this schedule takes 47. Against a reduction in every stage: P3 of
// 128 products 1450 -> 1418, P4 961 -> 949, P7 503 -> 485 us; 48 rotations 3.44 ->
// 3.40 ms.
struct IntAr {
    using T = u64;
    u64 q, two_q;
    __host__ __device__ static constexpr int fwd_out(int, int) { return 0; }
    __host__ __device__ static constexpr int inv_out(int, int) { return 0; }
    __device__ __forceinline__ u64 in(u64 x) const { return x; }
    __device__ __forceinline__ u64 in_canon(u64 x) const { return x; }
    __device__ __forceinline__ u64 bits(u64 x) const { return x; }
    __device__ __forceinline__ u64 unbits(u64 b) const { return b; }
    // lazy [0, 8q) -> canonical [0, q), or -> [0, 2q)
    __device__ __forceinline__ u64 final_2q(u64 b) const { return csub(csub(b, 2 * two_q), two_q); }
    __device__ __forceinline__ u64 final_canon(u64 b) const { return csub(final_2q(b), q); }
    template <int K, int L, class TW>
    __device__ __forceinline__ void ct_stage(u64 (&v)[1 << K], const TW& tw, u32 B) const {
        constexpr int half = 1 << (K - 1 - L);
#pragma unroll
        for (int g = 0; g < (1 << L); ++g) {
            const Tw t = tw((B << L) + g);
#pragma unroll
            for (int o = 0; o < half; ++o) {
                u64& x = v[g * 2 * half + o];
                u64& y = v[g * 2 * half + o + half];
                const u64 xx = int_ct_reduces(L) ? csub(x, 2 * two_q) : x;
                const u64 r = shoup_lazy(y, t.w, t.wp, q);
                x = xx + r;
                y = xx - r + two_q;
            }
        }
        if constexpr (L + 1 < K) ct_stage<K, L + 1>(v, tw, B);
    }
    template <int K, int L, class TW>
    __device__ __forceinline__ void gs_stage(u64 (&v)[1 << K], const TW& tw, u32 B) const {
        constexpr int s = K - 1 - L, half = 1 << s;
#pragma unroll
        for (int g = 0; g < (1 << L); ++g) {
            const Tw t = tw((B << L) + g);
#pragma unroll
            for (int o = 0; o < half; ++o) {
                const int i = g * 2 * half + o;
                u64& x = v[i];
                u64& y = v[i + half];
                const bool sums = int_gs_sums(s, o);   // both below 4q, else 2q
                const u64 d = x - y + (sums ? 2 * two_q : two_q);
                x = sums ? csub(x + y, 2 * two_q) : x + y;
                y = shoup_lazy(d, t.w, t.wp, q);
            }
        }
        if constexpr (L > 0) {
            gs_stage<K, L - 1>(v, tw, B);
        } else {
#pragma unroll
            for (int u = 0; u < half; ++u) v[u] = csub(v[u], two_q);   // the sums of the last stage
        }
    }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void fwd(u64 (&v)[1 << K], const TW& tw, u32 B) const { ct_stage<K, 0>(v, tw, B); }
    template <int K, int BIN, bool END, class TW>
    __device__ __forceinline__ void inv(u64 (&v)[1 << K], const TW& tw, u32 B) const { gs_stage<K, K - 1>(v, tw, B); }
};

// Geometry of the two passes for one LOGN. W: columns of the column pass's
// tile at 256 rows, COL_WIDE or COL_NARROW (half the threads per CTA and twice
// the CTAs, for grids that leave SMs idle; see narrow_tiles).
constexpr int COL_WIDE = 16, COL_NARROW = 8;
template <int LOGN, int W = COL_WIDE>
struct Geo {
    static_assert(LOGN >= 9 && LOGN <= 16, "LOGN out of range");
    static constexpr int N = 1 << LOGN;
    static constexpr int A = LOGN - 8;               // column stages
    static constexpr int R1 = 1 << A;                // rows
    static constexpr int COLS = 256;
    // column pass: all rows x C columns, <= 256 W elements, >= W columns
    static constexpr int C = cmin(256, cmax(W, (256 * W) >> A));
    static constexpr int COL_MINB = 64 / W;
    static constexpr int COL_TILE = R1 * C;
    static constexpr int COL_TILES = COLS / C;
    static constexpr int COL_THREADS = COL_TILE / 16;
    // row pass: RB rows x 256 (padded rows in shared memory). Warps own their
    // rows (below), so the CTA only sets how finely a small grid spreads: eight
    // rows, eight CTAs per SM, against sixteen rows and four: one product at
    // N = 2^15 110.0 -> 107.4 us, 128 products unchanged; four rows gave 106.6
    // and 437 instead of 434 us for 13 mixed operations at N = 2^14.
    static constexpr int RB = cmin(R1, 8);
    static constexpr int ROW_MINB = 8;
    static constexpr int ROW_TILE = RB * COLS;
    static constexpr int ROW_TILES = R1 / RB;
    static constexpr int ROW_THREADS = ROW_TILE / 16;
    static constexpr int ROW_STRIDE = COLS + COLS / 16;      // one pad word per 16
    static constexpr int COL_SMEM = COL_TILE * 8;
    static constexpr int ROW_SMEM = RB * ROW_STRIDE * 8;
};

// Column tiles of eight columns where sixteen would make at most two waves (of
// four CTAs per SM): one product (N = 2^15, 16-64 wide tiles a kernel) 89 -> 83 us,
// a transform of 3 + 3 rotations (N = 2^13, 24-726) 365 -> 356 us. On grids of
// many waves their 64-byte row segments cost more than they spread: 128 products
// 6.84 -> 7.03 ms with narrow tiles throughout.
template <int LOGN>
inline bool narrow_tiles(unsigned jobs, int sms) {
    return jobs * (unsigned)Geo<LOGN>::COL_TILES <= 8u * (unsigned)sms;
}

__device__ __forceinline__ int rowpad(int c) { return c + (c >> 4); }

// ------------------------------------------------------------------ column pass
// Round (J0, K) over a column tile: thread groups index gi -> (cl, lo, hidx).
// LD(r, cl) -> T and ST(r, cl, v) address tile-local column cl, global row r.
template <int A, int C, int NT, int J0, int K, bool FWD, int BIN, bool END, class AR, class TW, class LD, class ST>
__device__ __forceinline__ void col_round(const AR& ar, const TW& tw, LD&& ld, ST&& st) {
    constexpr int SH = A - J0 - K;
    constexpr int GROUPS = ((1 << A) * C) >> K;
    static_assert(GROUPS % NT == 0, "groups must divide evenly");
#pragma unroll 1
    for (int gi = threadIdx.x; gi < GROUPS; gi += NT) {
        const int cl = gi % C;
        const int rest = gi / C;
        const int lo = rest & ((1 << SH) - 1);
        const int hidx = rest >> SH;
        const int hi = hidx << (A - J0);
        typename AR::T v[1 << K];
#pragma unroll
        for (int u = 0; u < (1 << K); ++u) v[u] = ld(hi + (u << SH) + lo, cl);
        const u32 B = (1u << J0) + (u32)hidx;
        if constexpr (FWD) ar.template fwd<K, BIN, END>(v, tw, B);
        else ar.template inv<K, BIN, END>(v, tw, B);
#pragma unroll
        for (int u = 0; u < (1 << K); ++u) st(hi + (u << SH) + lo, cl, v[u]);
    }
}

// Barrier between rounds: the whole CTA by default; a warp-specialised
// kernel passes a named barrier over its transform warps.
struct CtaSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

// Forward column pass: stages 0..A-1. The first round reads the policy's
// values (bounded by BIN) through `ld`; the last stores the policy's own
// words (ar.bits) through `st`, for a following row pass; the rounds between
// go through shared memory `sm`.
template <int A, int C, int NT, int J0, int BIN, class AR, class TW, class LD, class ST, class SY = CtaSync>
__device__ __forceinline__ void fwd_col_rounds(u64* sm, const TW& tw, const AR& ar, LD&& ld, ST&& st,
                                               const SY& sync = SY{}) {
    constexpr int K = cmin(4, A - J0);
    constexpr bool FIRST = (J0 == 0);
    constexpr bool LAST = (J0 + K == A);
    using T = typename AR::T;
    auto gst = [&](int r, int cl, T v) { st(r, cl, ar.bits(v)); };
    auto sld = [&](int r, int cl) { return ar.unbits(sm[r * C + cl]); };
    auto sst = [&](int r, int cl, T v) { sm[r * C + cl] = ar.bits(v); };
    if constexpr (FIRST && LAST) col_round<A, C, NT, J0, K, true, BIN, false>(ar, tw, ld, gst);
    else if constexpr (FIRST) col_round<A, C, NT, J0, K, true, BIN, false>(ar, tw, ld, sst);
    else if constexpr (LAST) col_round<A, C, NT, J0, K, true, BIN, false>(ar, tw, sld, gst);
    else col_round<A, C, NT, J0, K, true, BIN, false>(ar, tw, sld, sst);
    if constexpr (!LAST) {
        sync();
        fwd_col_rounds<A, C, NT, J0 + K, AR::fwd_out(K, BIN)>(sm, tw, ar, ld, st, sync);
    }
}

// Inverse column pass: stages A-1..0 (GS). Rounds run from the top stage
// group down; JE is the exclusive end of the current round's stage range.
// `ld` returns the words of an inverse row pass as the policy's values
// (bounded by BIN); `st` receives the policy's values (IntAr: [0, 2q);
// FpArS: below 8q).
template <int A, int C, int NT, int JE, int BIN, class AR, class TW, class LD, class ST>
__device__ __forceinline__ void inv_col_rounds(u64* sm, const TW& tw, const AR& ar, LD&& ld, ST&& st) {
    // partition identical to the forward one: rounds [0,4),[4,8),... last ragged
    constexpr int J0 = ((JE - 1) / 4) * 4;
    constexpr int K = JE - J0;
    constexpr bool FIRST = (JE == A);
    constexpr bool LAST = (J0 == 0);
    using T = typename AR::T;
    auto sld = [&](int r, int cl) { return ar.unbits(sm[r * C + cl]); };
    auto sst = [&](int r, int cl, T v) { sm[r * C + cl] = ar.bits(v); };
    if constexpr (FIRST && LAST) col_round<A, C, NT, J0, K, false, BIN, true>(ar, tw, ld, st);
    else if constexpr (FIRST) col_round<A, C, NT, J0, K, false, BIN, false>(ar, tw, ld, sst);
    else if constexpr (LAST) col_round<A, C, NT, J0, K, false, BIN, true>(ar, tw, sld, st);
    else col_round<A, C, NT, J0, K, false, BIN, false>(ar, tw, sld, sst);
    if constexpr (!LAST) {
        __syncthreads();
        inv_col_rounds<A, C, NT, J0, AR::inv_out(K, BIN)>(sm, tw, ar, ld, st);
    }
}

// ------------------------------------------------------------------ row pass
// Round (J0, K) over a row tile of RB rows; global row of tile row 0 is R0.
// Twiddle base B = 2^(A+J0) + ((R0+rl) << J0) + hidx. Thread t works on row
// t / 16 in every round and in the walks below, so a warp owns two rows from
// load to store and a row pass needs no barrier between warps: each runs
// ahead on its own, where a barrier per round had all eight wait for the last
// (1.1-1.6 barrier stalls per issue). Phases of 128 products with the barriers
// -> without: P1 336 -> 323, P4 1012 -> 959, P6 393 -> 363, P9 573 -> 541 us.
template <int A, int RB, int NT, int J0, int K, bool FWD, int BIN, bool END, class AR, class TW, class LD, class ST>
__device__ __forceinline__ void row_round(const AR& ar, const TW& tw, u32 R0, LD&& ld, ST&& st) {
    constexpr int SH = 8 - J0 - K;
    constexpr int GROUPS = (RB * 256) >> K;
    static_assert(GROUPS == NT && K == 4, "a thread owns one radix-16 group of its row in every round");
    const int gi = threadIdx.x;
    const int lo = gi & ((1 << SH) - 1);
    const int rest = gi >> SH;
    const int hidx = rest & ((1 << J0) - 1);
    const int rl = rest >> J0;
    const int cb = (hidx << (8 - J0)) + lo;
    typename AR::T v[1 << K];
#pragma unroll
    for (int u = 0; u < (1 << K); ++u) v[u] = ld(rl, cb + (u << SH));
    const u32 B = (1u << (A + J0)) + ((R0 + (u32)rl) << J0) + (u32)hidx;
    if constexpr (FWD) ar.template fwd<K, BIN, END>(v, tw, B);
    else ar.template inv<K, BIN, END>(v, tw, B);
#pragma unroll
    for (int u = 0; u < (1 << K); ++u) st(rl, cb + (u << SH), v[u]);
}

// Forward row pass: stages A..A+7, two rounds of four. The first round reads a
// forward column pass's words as the policy's values (bounded by BIN) with
// `ld` directly; the last round writes shared memory, and the caller then
// reads the tile row-contiguously (coalesced) and converts each word with
// ar.final_canon or ar.final_2q.
template <int A, int RB, int NT, int J0, int BIN, class AR, class TW, class LD>
__device__ __forceinline__ void fwd_row_rounds(u64* sm, const TW& tw, u32 R0, const AR& ar, LD&& ld) {
    constexpr int K = 4;
    constexpr bool LAST = (J0 + K == 8);
    constexpr int STR = 256 + 16;
    using T = typename AR::T;
    auto sld = [&](int rl, int c) { return ar.unbits(sm[rl * STR + rowpad(c)]); };
    auto sst = [&](int rl, int c, T v) { sm[rl * STR + rowpad(c)] = ar.bits(v); };
    if constexpr (J0 == 0) row_round<A, RB, NT, J0, K, true, BIN, LAST>(ar, tw, R0, ld, sst);
    else row_round<A, RB, NT, J0, K, true, BIN, LAST>(ar, tw, R0, sld, sst);
    __syncwarp();
    if constexpr (!LAST) fwd_row_rounds<A, RB, NT, J0 + K, AR::fwd_out(K, BIN)>(sm, tw, R0, ar, ld);
}

// Inverse row pass: GS stages A+7..A. Input is staged into shared memory
// (row-contiguous, coalesced) by the caller as the policy's words (bounded by
// BIN); the last round stores the policy's own words via `st`, for a
// following column pass.
template <int A, int RB, int NT, int JE, int BIN, class AR, class TW, class ST>
__device__ __forceinline__ void inv_row_rounds(u64* sm, const TW& tw, u32 R0, const AR& ar, ST&& st) {
    constexpr int K = 4, J0 = JE - K;
    constexpr bool LAST = (J0 == 0);
    constexpr int STR = 256 + 16;
    using T = typename AR::T;
    auto gst = [&](int rl, int c, T v) { st(rl, c, ar.bits(v)); };
    auto sld = [&](int rl, int c) { return ar.unbits(sm[rl * STR + rowpad(c)]); };
    auto sst = [&](int rl, int c, T v) { sm[rl * STR + rowpad(c)] = ar.bits(v); };
    if constexpr (LAST) row_round<A, RB, NT, J0, K, false, BIN, false>(ar, tw, R0, sld, gst);
    else {
        row_round<A, RB, NT, J0, K, false, BIN, false>(ar, tw, R0, sld, sst);
        __syncwarp();
        inv_row_rounds<A, RB, NT, J0, AR::inv_out(K, BIN)>(sm, tw, R0, ar, st);
    }
}

// Coalesced walks over a row tile, each warp over its own two rows (16 words
// per thread, a warp touching 256 contiguous bytes per step): word e of the
// tile lies at padded shared-memory index si; both advance by constants from
// the thread's first word.
template <int RB, int NT, class F>
__device__ __forceinline__ void row_tile_walk(F&& f) {
    static_assert(NT == RB * 16, "two rows per warp");
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int e0 = w * 512 + l, s0 = w * 2 * (256 + 16) + rowpad(l);
#pragma unroll
    for (int k = 0; k < 16; ++k) f(e0 + k * 32, s0 + (k / 8) * (256 + 16) + rowpad(k % 8 * 32));
}

// Same walk for staging a tile: every load of the thread is issued before the
// first conversion and shared-memory store.
template <int RB, int NT, class LD, class ST>
__device__ __forceinline__ void row_tile_stage(LD&& ld, ST&& st) {
    u64 v[16];
    int k = 0;
    row_tile_walk<RB, NT>([&](int e, int) { v[k++] = ld(e); });
    k = 0;
    row_tile_walk<RB, NT>([&](int e, int si) { st(e, si, v[k++]); });
}

// Two-operand staging in batches of 8 words per thread: both operands of a
// batch are loaded before st(e, si, a, b) combines them.
template <int RB, int NT, class LDA, class LDB, class ST>
__device__ __forceinline__ void row_tile_stage2(LDA&& lda, LDB&& ldb, ST&& st) {
    constexpr int BT = 8;
    u64 a[BT], b[BT];
    int k = 0;
    row_tile_walk<RB, NT>([&](int e, int si) {
        if (k % BT == 0) {
#pragma unroll
            for (int j = 0; j < BT; ++j) {
                a[j] = lda(e + j * 32);
                b[j] = ldb(e + j * 32);
            }
        }
        st(e, si, a[k % BT], b[k % BT]);
        ++k;
    });
}

}  // namespace ntt
