// Basis conversion into a tower q < 2^50 by an FP64 quotient: the rule that
// admits it, its constants and its arithmetic. Compiles as plain C++ too, so
// that the CPU check runs the functions that the kernels (P8 in pipeline.cuh)
// compile in.
//
// sum_t x_t c_t mod q needs only
//   r1 = sum_t x_t c_t - K q   (mod 2^64),   K near S = sum_t x_t (c_t / q),
// as long as r1 fits 64 bits: low 64-bit products on the integer pipes (one
// wide and two narrow multiplies) and one FMA per term for S on the FP64 pipe.
// Constants are signed, |c_t / q| <= 1/2. Sources below 2^b are rounded to
// doubles, so S sums n terms with an error of at most 2^(b-54) (n (n+1) / 2 +
// 5 n / 2); K is S rounded to a multiple of 2^12 (error 2^11). Where
// conv_wrap_ok admits (n, b), |r1| < 8000 q < 2^63. A second step subtracts K2 q,
// K2 the integer nearest to RN(r1) RN(1/q): the two roundings move that
// quotient by at most 2^13 (2^-53 + 2^-53) = 2^-39, so |r| <= (1/2 + 2^-39) q,
// inside the normalised bound (B_NORM, q/2 + q/512) that the transform takes.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#include "fp_sched.hpp"

namespace gfx {

// Whether a conversion of n sources below `below` (2^b) into a tower below 2^50
// may take the FP64-quotient form: the quotient's error, in units, times q has
// to stay below 2^63. Ten sources at 60 bits, seven at 61.
constexpr bool conv_wrap_ok(unsigned n, uint64_t below) {
    int b = 0;
    while (b < 63 && (1ull << b) < below) ++b;
    double unit = 1.0;   // 2^(b - 54)
    for (int k = 54; k < b; ++k) unit *= 2.0;
    for (int k = b; k < 54; ++k) unit *= 0.5;
    return b <= 61 && unit * (0.5 * n * (n + 1) + 2.5 * n) + 2048.0 + 64.0 < 8000.0;
}

}  // namespace gfx

namespace pl {

// One term of a basis conversion: the constant, and its ratio to the target
// modulus (quotient form) or its value as a double (P3's FP64 products).
struct alignas(16) ConvTerm { uint64_t c; double f; };

// The IEEE operations of the quotient form.
GFX_HD inline double q_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
GFX_HD inline double q_add(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
GFX_HD inline double q_mul(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
GFX_HD inline long long q_bits(double x) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(x);
#else
    long long v;
    std::memcpy(&v, &x, 8);
    return v;
#endif
}
GFX_HD inline double q_double(long long x) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(x);
#else
    double v;
    std::memcpy(&v, &x, 8);
    return v;
#endif
}

// The term of the residue c (canonical mod q), negated when NEG.
template <bool NEG>
GFX_HD inline ConvTerm conv_term(uint64_t c, uint64_t q, double qinv) {
    long long v = c > (q >> 1) ? (long long)c - (long long)q : (long long)c;
    if (NEG) v = -v;
    return ConvTerm{(uint64_t)v, q_mul((double)v, qinv)};
}
// lo += x c mod 2^64, s += x c / q. Words become doubles by the conversion
// instruction: two FP64 additions of biased halves took four issue slots (P8 of
// 128 products 960 -> 912 us).
GFX_HD inline void quot_term(uint64_t& lo, double& s, uint64_t x, const ConvTerm& t) {
    lo += x * t.c;
    s = q_fma((double)x, t.f, s);
}
struct WrapConv {
    uint64_t q;
    double qinv;
    // r = lo - K q - K2 q, |r| <= (1/2 + 2^-39) q
    GFX_HD long long finish(uint64_t lo, double s) const {
        const long long k = q_bits(q_add(s, 0x1.8p64)) - 0x43F8000000000000ll;
        const uint64_t r1 = lo - (uint64_t)k * (q << 12);
        const double rd = (double)(long long)r1;
        const int k2 = (int)(uint32_t)(uint64_t)q_bits(q_fma(rd, qinv, ntt::FP_M1));
        return (long long)(r1 - (uint64_t)(long long)k2 * q);
    }
    GFX_HD double finish_d(uint64_t lo, double s) const {
        return q_add(q_double(finish(lo, s) + 0x4338000000000000ll), -ntt::FP_M1);
    }
};

}  // namespace pl
