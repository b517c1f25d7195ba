// Exact modular arithmetic for odd primes p < 2^50 in double precision.
//
// A residue is a double holding a whole number x with |x| <= a p for a small bound a (values are
// signed and not canonical; every function states its bounds in multiples of p).  The product of
// two residues takes six double-precision operations, all of which issue at 64 per SM per clock on
// B200 (a butterfly takes eight), where a 64-bit Shoup product takes nine 32-bit multiplies of the same
// rate and about as many adds.  n = 16384, 148 primes: 66.6 primes a second with integers, 148 this way.
// The product is the one of van der Hoeven, Lecerf and Quintin, "Modular SIMD arithmetic in Mathemagix"
// (2016): the high part of x w, its error by an FMA, a rounded quotient and its remainder.
//
// Why it is exact (p < 2^50, |x w| <= 2^51 p):
//   h = fl(x w); x w = h + l with l = fma(x, w, -h) exact (an FMA's rounding error of a product).
//   q = the whole number nearest fl(h fl(1/p)): adding and subtracting 1.5 2^52 rounds to a whole
//     number while |x w / p| <= 2^51.  h and 1/p are each within 2^-53 relative, so
//     |q - x w / p| <= 1/2 + |x w / p| 2^-52.
//   h - q p is a whole number (h is a multiple of its unit in the last place, which is one or
//     more when h is not exact, and q p is whole) of size below 2^53, so the FMA that forms it is exact, and
//     so is the sum with l.  The result is x w - q p.
#pragma once
#include <cmath>
#include <cstring>

#include "modarith.cuh"

namespace cfb {

#if defined(__CUDA_ARCH__)
CF_HD double fp_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
CF_HD double fp_mul(double a, double b) { return __dmul_rn(a, b); }
CF_HD double fp_add(double a, double b) { return __dadd_rn(a, b); }
CF_HD double fp_bits(u64 w) { return __longlong_as_double((long long)w); }
CF_HD u64 fp_word(double x) { return (u64)__double_as_longlong(x); }
CF_HD long long fp_whole(double x) { return __double2ll_rn(x); }
#else
inline double fp_fma(double a, double b, double c) { return std::fma(a, b, c); }
inline double fp_mul(double a, double b) { return a * b; }
inline double fp_add(double a, double b) { return a + b; }
inline double fp_bits(u64 w) {
    double x;
    std::memcpy(&x, &w, 8);
    return x;
}
inline u64 fp_word(double x) {
    u64 w;
    std::memcpy(&w, &x, 8);
    return w;
}
inline long long fp_whole(double x) { return (long long)x; }
#endif

struct FpMod {
    double p, pinv;  // the prime and fl(1/p)
};

// x w mod p: |result| <= (1/2 + a b / 4) p for |x| <= a p, |w| <= b p, a b <= 2
CF_HD double fp_mulmod(double x, double w, const FpMod& m) {
    constexpr double M = 6755399441055744.0;  // 1.5 2^52
    const double h = fp_mul(x, w);
    const double q = fp_add(fp_fma(h, m.pinv, M), -M);
    const double l = fp_fma(x, w, -h);
    return fp_add(fp_fma(-q, m.p, h), l);
}
// x mod p: |result| <= 0.51 p for |x| <= 8 p
CF_HD double fp_red(double x, const FpMod& m) {
    constexpr double M = 6755399441055744.0;
    const double q = fp_add(fp_fma(x, m.pinv, M), -M);
    return fp_fma(-q, m.p, x);
}
// the canonical residue of x, |x| <= 8 p, as an integer
CF_HD u64 fp_canon(double x, const FpMod& m) {
    const long long v = fp_whole(fp_red(x, m));
    return v < 0 ? (u64)(v + (long long)m.p) : (u64)v;
}
// a canonical residue as a double, centred: |result| <= p / 2
CF_HD double fp_centre(u64 v, u64 p) { return v > p / 2 ? -(double)(long long)(p - v) : (double)(long long)v; }
// x^e for |x| <= 0.75 p: |result| <= 0.75 p
CF_HD double fp_pow(double x, u64 e, const FpMod& m) {
    double r = 1.0;
    while (e) {
        if (e & 1) r = fp_mulmod(r, x, m);
        e >>= 1;
        if (e) x = fp_mulmod(x, x, m);
    }
    return r;
}
// x^k, |x| <= 0.75 p: each turn's two products are independent, so the chain is one product per bit of k
CF_HD double fp_pow_fast(double x, int k, const FpMod& m) {
    double r = 1.0;
#pragma unroll 1
    for (; k; k >>= 1) {
        const double y = fp_mulmod(r, x, m);
        r = k & 1 ? y : r;
        x = fp_mulmod(x, x, m);
    }
    return r;
}

}  // namespace cfb
