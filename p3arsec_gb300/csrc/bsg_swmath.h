// bsg_swmath.h -- the elementary functions of the swaption Monte Carlo, in
// 64-bit fixed point: the normal variates (Box-Muller from the bits of the
// uniforms) and the powers of two of the discount factors; and a
// double-precision exp for rates outside the fixed-point range.
//
// Why fixed point: GB300 issues 2 double-precision operations per clock and
// SM against 32 32x32->64-bit integer multiply-adds and 64-128 other integer
// operations (measured), so a 64-bit product truncated to its high half
// (three multiply-adds) costs a fifth of a double multiply and carries 11
// more bits, and the high-order terms of a series fit 32 bits at a thirtieth
// of the cost.  Every value here has at least 57 fraction bits; a normal
// variate is within 2e-17 + half an ulp of the exact one.
//
// The uniforms are u = (2k + 1) 2^-53 for a 52-bit integer k (the grid of
// midpoints in (0, 1)); a pair (u1, u2) gives z0 = sqrt(-2 ln u1) cos(2 pi u2)
// and z1 = sqrt(-2 ln u1) sin(2 pi u2).  Both functions start from k itself,
// so neither the uniform nor the angle is ever rounded:
//
//  -2 ln u: u = 2^e m with m in [1, 2) read off k's bits; c (20 bits) is the
//    reciprocal of the middle of m's 1/512 interval, m c = 1 + r exactly
//    (|r| < 2^-10), -2 ln u = -2 e ln 2 + 2 ln c - 2 ln(1 + r) with ln(1 + r)
//    by its Taylor series to r^6.  For m >= 1.5 the table holds ln(2 c) and e
//    is one larger, so that u near 1 (e = -1, c = 1/2) gives -2 ln(1 + r)
//    alone, as small as it is, from a normalised r.  This is the table-driven
//    logarithm of P. T. P. Tang, ACM TOMS 16(4), 1990, with the reciprocal
//    table's exact products.
//  sqrt: a linear table seed at or below 1/sqrt(y) (192 intervals), then
//    s = y y0 (1 + e/2 + 3 e^2/8), e = 1 - y y0^2 < 2^-14 (the binomial series
//    of (1 - e)^(-1/2); its cubic term, folded into the quadratic's factor).
//  sin/cos(2 pi u): the quadrant and the nearest 1/1024 turn of u from k's
//    bits, the rest an exact integer; the angle-addition formulas combine the
//    table's sin and cos with Taylor polynomials of sin phi (to phi^5) and
//    1 - cos phi (to phi^6), |phi| <= pi/1024.
//  2^x: the integer part, a table of 2^(j/1024), and the Taylor polynomial of
//    e^t - 1 to t^4, t = r ln 2 < 2^-10.
//  e^x (double): x = (64 m + j) ln2/64 + r with k = 64 m + j the integer
//    nearest 64 x / ln 2 (|r| <= ln2/128), e^x = 2^m 2^(j/64) (1 + p(r)), p the
//    Taylor polynomial of e^r - 1 to r^6; ln2/64 in two parts so that r is
//    exact to far below its ulp (P. T. P. Tang, ACM TOMS 15(2), 1989).
//    Arguments of magnitude 700 or more (and NaN) go to the platform's exp.
//
// Everything is integer work or an explicitly rounded IEEE operation, so the
// host build of this header (compile it with -ffp-contract=off) gives the
// same bits as the GPU; the CPU test checks the very code the GPU runs.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "bsg_swmath_tables.h"

#if defined(__CUDACC__)
#define BSG_SW_FN __host__ __device__ __forceinline__
#else
#define BSG_SW_FN inline
#endif

namespace bsg_sw {

struct alignas(16) LogEntry { int64_t ln; uint32_t c; };
struct alignas(8) SeedEntry { uint32_t a, b; };
struct alignas(16) Angle { uint64_t s, c; };

// 22,528 bytes: the kernels copy it into shared memory once per block.
struct alignas(16) Tables {
    LogEntry lg[512];
    SeedEntry rs[192];  // y in [i/256, (i + 1)/256), i = 64..255
    Angle ang[256];     // the first quadrant
    uint64_t e2[1024];  // 2^(j/1024)
    double e64[64];     // 2^(j/64)
};

#if defined(__CUDA_ARCH__)
BSG_SW_FN double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
BSG_SW_FN double mul(double a, double b) { return __dmul_rn(a, b); }
BSG_SW_FN double add(double a, double b) { return __dadd_rn(a, b); }
BSG_SW_FN double from_bits(uint64_t u) { return __longlong_as_double((long long)u); }
BSG_SW_FN int clz64(uint64_t v) { return __clzll((long long)v); }
BSG_SW_FN uint64_t to_bits(double d) { return (uint64_t)__double_as_longlong(d); }
BSG_SW_FN double exp_fallback(double x) { return exp(x); }
BSG_SW_FN uint32_t hi32x32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
BSG_SW_FN int32_t shi32x32(int32_t a, int32_t b) { return __mulhi(a, b); }
#else
inline double fma_(double a, double b, double c) { return fma(a, b, c); }
inline double mul(double a, double b) { return a * b; }
inline double add(double a, double b) { return a + b; }
inline double from_bits(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
inline int clz64(uint64_t v) { return __builtin_clzll(v); }
inline uint64_t to_bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
inline double exp_fallback(double x) { return exp(x); }
inline uint32_t hi32x32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline int32_t shi32x32(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
#endif

BSG_SW_FN uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
BSG_SW_FN uint32_t hi32(uint64_t a) { return (uint32_t)(a >> 32); }
// The high half of a 64x64-bit product without its lowest partial product:
// at most 2 units below the exact one.
BSG_SW_FN uint64_t mulhi(uint64_t a, uint64_t b) {
    const uint64_t cross = (uint64_t)hi32x32(hi32(a), (uint32_t)b) + hi32x32((uint32_t)a, hi32(b));
    return wide(hi32(a), hi32(b)) + cross;
}
// a b / 2^32, at most 1 unit below.
BSG_SW_FN uint64_t mul_64x32(uint64_t a, uint32_t b) {
    return wide(hi32(a), b) + hi32x32((uint32_t)a, b);
}

// The 52-bit integer k of a uniform from two 32-bit random words (the top
// 20 bits of a, all of b).
BSG_SW_FN uint64_t unit_bits(uint32_t a, uint32_t b) { return ((uint64_t)(a >> 12) << 32) | b; }

// -2 ln u for u = (2k + 1) 2^-53, k < 2^52, as x 2^-s with x's top bit set.
struct Scaled { uint64_t x; int s; };

BSG_SW_FN Scaled neg2_ln_scaled(const Tables& t, uint64_t k) {
    const uint64_t v = 2 * k + 1;                        // u = v 2^-53, v odd
    const int lz = clz64(v);                             // 11..63
    const uint64_t m = v << lz;                          // u = (m 2^-63) 2^(10 - lz)
    const int i = (int)((m >> 54) & 511);
    const LogEntry le = t.lg[i];
    const int ne = lz - 10 - (i >> 8);                   // powers of two taken out, negated: 0..53
    // r 2^73, exact: m c 2^20 - 2^83 (a multiple of 2^73 times 2^10, mod 2^64 after the shift)
    const uint64_t lo = wide((uint32_t)m, le.c);
    const uint64_t hi = wide(hi32(m), le.c) + (lo >> 32);
    const int64_t r = (int64_t)((hi << 22) | ((uint32_t)lo >> 10));
    const int32_t rh = (int32_t)(r >> 32);               // r 2^41
    // -2 ln(1 + r) = -2 r + r^2 q, q = 1 - r (2/3 - r (1/2 - r (2/5 - r/3)))
    int32_t q = 858993459 - (shi32x32(rh, 715827883) >> 9);  // 2/5 - r/3, 31 fraction bits
    q = 1073741824 - (shi32x32(rh, q) >> 9);
    q = 1431655765 - (shi32x32(rh, q) >> 9);
    const uint64_t q63 = (1ull << 63) - (uint64_t)(((int64_t)rh * q) >> 9);
    if (ne == 0 && i == 511) {
        // u near 1: -2 ln u = 2 |r| (1 + c), c = |r|/2 + r^2/3 + |r|^3/4 + r^4/5,
        // from |r| = 1 - u (2^-53 and up) with its top bit moved up
        const uint64_t ar = 0ull - (uint64_t)r;          // |r| 2^73
        const uint32_t ah = hi32(ar);                    // 41
        const uint64_t a2 = wide(ah, ah) + ((uint64_t)hi32x32(ah, (uint32_t)ar) << 1);  // r^2, 82
        const uint32_t g = hi32x32(ah, 1073741824u + (hi32x32(ah, 858993459u) >> 9));   // |r| (1/4 + |r|/5), 41
        const uint64_t c = (ar >> 10) + (mulhi(a2, 6148914691236517205ull) >> 18) +
                           (wide(hi32(a2), g) >> 27);    // 64
        const int n = clz64(ar);
        const uint64_t arn = (ar << n) >> 1;
        const uint64_t y = arn + mulhi(arn, c);          // below 2^63 (1 + 2^-11): may carry
        const int top = (int)(y >> 63);
        return {y << (1 - top), n + 72 - top};
    }
    // r^2 2^82, the cross term rounded down by at most 4: + 4 keeps it positive
    const uint64_t r2 = (uint64_t)((int64_t)rh * rh + 4) +
                        (uint64_t)((int64_t)shi32x32(rh, (int32_t)((uint32_t)r >> 1)) * 4);
    const uint64_t w = (uint64_t)le.ln + (mulhi(r2, q63) >> 19) - (uint64_t)(r >> 10);      // 62 bits
    // below 2 at ne = 0, where it may be small; below 73.5 otherwise
    const uint64_t x = ne == 0 ? w
                               : (uint64_t)((int64_t)w >> 5) + wide((uint32_t)BSG_SW_2LN2_57, (uint32_t)ne) +
                                     (wide(hi32(BSG_SW_2LN2_57), (uint32_t)ne) << 32);
    const int n = clz64(x);
    return {x << n, (ne == 0 ? 62 : 57) + n};
}

BSG_SW_FN double scaled_to_double(uint64_t x, int s) {   // x 2^-s, x's top bit set
    const uint64_t m = (x >> 11) + ((x >> 10) & 1);      // 2^52..2^53: the leading bit adds 1 to the exponent
    return from_bits(m + ((uint64_t)(1022 + 63 - s) << 52));
}

// -2 ln u as a double: a value in (0, 73.5].
BSG_SW_FN double neg2_ln_unit(const Tables& t, uint64_t k) {
    const Scaled w = neg2_ln_scaled(t, k);
    return scaled_to_double(w.x, w.s);
}

// sqrt(x 2^-w.s) = s 2^(e - 62), s in [2^61, 2^62].
struct Root { uint64_t s; int e; };

BSG_SW_FN Root sqrt_scaled(const Tables& t, Scaled w) {
    const int b = 64 - w.s;                              // the value is (x 2^-64) 2^b
    const int odd = b & 1;
    const uint64_t y = w.x >> odd;                       // [1/4, 1), 64 fraction bits
    const SeedEntry se = t.rs[(int)(y >> 56) - 64];
    const uint32_t y0 = se.a - hi32x32(se.b, (uint32_t)(y >> 24));  // 30 bits, at or below 1/sqrt(y)
    const uint64_t e = (1ull << 60) - mulhi(y, wide(y0, y0));       // 1 - y y0^2 in [0, 2^-14), 60 bits
    const uint32_t eh = (uint32_t)(e >> 14);             // e 2^46
    const uint32_t g = 805306368u + (hi32x32(eh, 671088640u) >> 14);  // 3/8 + 5/16 e, 31 bits
    const uint64_t corr = (e >> 1) + ((uint64_t)hi32x32(hi32(wide(eh, eh)), g) << 1);  // 60 bits
    const uint64_t s0 = mul_64x32(y, y0);                // 62 bits
    return {s0 + (mulhi(s0, corr << 17) >> 13), (b + odd) / 2};
}

// |sin| and |cos| of 2 pi u (u = (2k + 1) 2^-53) with 63 fraction bits up to
// the quadrant: in quadrant q (0..3) the angle is q quarter turns past the
// one whose sine and cosine these are.  Both may be off the first quadrant by
// half a table step, so they are signed: 62 fraction bits.
BSG_SW_FN void sincos_quadrant(const Tables& t, uint64_t k, int* quadrant, int64_t* s, int64_t* c) {
    const uint32_t j = (uint32_t)((k + (1ull << 41)) >> 42);  // nearest 1/1024: 0..1024
    const int64_t x = (int64_t)(2 * k + 1) - ((int64_t)j << 43);  // odd, |x| < 2^42
    const uint64_t neg = (uint64_t)(x >> 63);
    const uint64_t ax = ((uint64_t)x ^ neg) - neg;
    const uint64_t ph = mulhi(ax << 22, BSG_SW_2PI_61);  // |phi| = |x| 2 pi 2^-53, 72 fraction bits
    const uint32_t phh = hi32(ph);                       // 40
    const uint64_t p = wide(phh, phh) + ((uint64_t)hi32x32(phh, (uint32_t)ph) << 1);  // phi^2, 80
    const uint32_t pp = hi32(p);                         // 48
    // sin = phi - phi sg, sg = phi^2 (1/6 - phi^2/120)
    const uint32_t mu = 2863311531u - hi32x32(pp, 2185u);             // 34
    const uint32_t sg = (uint32_t)(wide(pp, mu) >> 31);               // 51
    const uint64_t sp = ph - (wide(phh, sg) >> 19);                   // 72
    // 1 - cos = phi^2 (1/2 - phi^2 (1/24 - phi^2/720))
    const uint32_t la = 2863311531u - hi32x32(pp, 1456u);             // 36
    const uint64_t ka = (1ull << 62) - (wide(pp, la) >> 21);          // 63
    const uint64_t cm = mulhi(p, ka);                                 // 79
    const Angle a = t.ang[j & 255];
    // a.s, a.c: 63 bits; products with sp: 71, with cm: 78
    const uint64_t csp = mulhi(a.c, sp) >> 9, ssp = mulhi(a.s, sp) >> 9;  // 62
    *s = (int64_t)((a.s >> 1) - (mulhi(a.s, cm) >> 16) + ((csp ^ neg) - neg));
    *c = (int64_t)((a.c >> 1) - (mulhi(a.c, cm) >> 16) - ((ssp ^ neg) - neg));
    *quadrant = (int)(j >> 8) & 3;
}

// cos and sin of 2 pi u with 62 fraction bits.
BSG_SW_FN void sincos_2pi_fixed(const Tables& t, uint64_t k, int64_t* s, int64_t* c) {
    int q;
    int64_t s1, c1;
    sincos_quadrant(t, k, &q, &s1, &c1);
    const int64_t ss = (q & 1) ? c1 : s1, cc = (q & 1) ? s1 : c1;
    *s = (q & 2) ? -ss : ss;
    *c = ((q + 1) & 2) ? -cc : cc;
}

// A 62-bit fixed-point value of magnitude at most 1 as a double.
BSG_SW_FN double fixed_to_double(int64_t a, int bits) {
    if (a == 0) return 0.0;
    const uint64_t neg = (uint64_t)(a >> 63), m = ((uint64_t)a ^ neg) - neg;
    const int n = clz64(m);
    return from_bits(to_bits(scaled_to_double(m << n, bits + n)) | (neg << 63));
}

BSG_SW_FN void sincos_2pi_unit(const Tables& t, uint64_t k, double* s, double* c) {
    int64_t sf, cf;
    sincos_2pi_fixed(t, k, &sf, &cf);
    *s = fixed_to_double(sf, 62);
    *c = fixed_to_double(cf, 62);
}

// r f, f in [-1, 1] with 62 fraction bits, as a fixed-point variate of 58
// fraction bits (|z| < 8.6).
constexpr int kZBits = 58;
BSG_SW_FN int64_t times_root(Root r, int64_t f) {
    const uint64_t neg = (uint64_t)(f >> 63), m = ((uint64_t)f ^ neg) - neg;
    const uint64_t z = mulhi(r.s << 1, m << 1) >> (4 - r.e);  // 62 + e bits before the shift, e <= 4
    return (int64_t)((z ^ neg) - neg);
}

// Normal variates z0, z1 (58 fraction bits) from four random words: u1 from
// (w0, w1), u2 from (w2, w3).  With BOTH false z1 is not computed.
template <bool BOTH>
BSG_SW_FN void normal_pair_fixed(const Tables& t, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3,
                                 int64_t* z0, int64_t* z1) {
    const Root r = sqrt_scaled(t, neg2_ln_scaled(t, unit_bits(w0, w1)));
    int64_t s, c;
    sincos_2pi_fixed(t, unit_bits(w2, w3), &s, &c);
    *z0 = times_root(r, c);
    if (BOTH) *z1 = times_root(r, s);
}

// The same as doubles.
BSG_SW_FN void normal_pair(const Tables& t, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3,
                           double* z0, double* z1) {
    int64_t a, b;
    normal_pair_fixed<true>(t, w0, w1, w2, w3, &a, &b);
    *z0 = fixed_to_double(a, kZBits);
    *z1 = fixed_to_double(b, kZBits);
}

// 2^(x 2^-57), |x 2^-57| < 64, as a double.
constexpr int kXBits = 57;
BSG_SW_FN double exp2_fixed(const Tables& t, int64_t x) {
    const uint64_t a = ((uint64_t)x & ((1ull << 47) - 1)) << 17;      // r < 2^-10, 74 fraction bits
    const uint64_t tt = mulhi(a, BSG_SW_LN2_64);                      // t = r ln 2, 74
    const uint32_t th = hi32(tt);                                     // 42
    const uint64_t t2 = wide(th, th) + ((uint64_t)hi32x32(th, (uint32_t)tt) << 1);  // t^2, 84
    const uint32_t g = 2863311531u + hi32x32(th, 699051u);            // 1/6 + t/24, 34
    const uint64_t t3g = wide(hi32(t2), hi32x32(th, g));              // t^3 g, 52 + 44 = 96
    const uint64_t p = tt + (t2 >> 11) + (t3g >> 22);                 // e^t - 1, 74
    const uint64_t e = t.e2[(x >> 47) & 1023];                        // 63
    const uint64_t y = e + (mulhi(e, p) >> 10);                       // [1, 2), 63
    return from_bits((y >> 11) + ((y >> 10) & 1) + ((uint64_t)(1022 + (x >> kXBits)) << 52));
}

// e^x; for |x| >= 700 or NaN, the platform's exp.
BSG_SW_FN double exp_(const Tables& t, double x) {
    if ((to_bits(x) & 0x7FFFFFFFFFFFFFFFull) >= 0x4085E00000000000ull) return exp_fallback(x);  // 700
    const double tm = fma_(x, BSG_SW_INV_L, 6755399441055744.0);  // 1.5 2^52 + k
    const double kd = add(tm, -6755399441055744.0);
    const int k = (int)(uint32_t)to_bits(tm);                      // |k| < 2^16
    double r = fma_(-kd, BSG_SW_L1, x);
    r = fma_(-kd, BSG_SW_L2, r);
    double q = 1.0 / 720;
    q = fma_(q, r, 1.0 / 120);
    q = fma_(q, r, 1.0 / 24);
    q = fma_(q, r, 1.0 / 6);
    q = fma_(q, r, 0.5);
    const double p = fma_(mul(r, r), q, r);                        // e^r - 1
    const double tj = t.e64[k & 63];
    const double y = fma_(tj, p, tj);                              // in [0.99, 2.01)
    return from_bits(to_bits(y) + ((uint64_t)(int64_t)(k >> 6) << 52));
}

}  // namespace bsg_sw

// The tables' initializer: `const bsg_sw::Tables t = BSG_SW_TABLES;`
#define BSG_SW_TABLES \
    {{BSG_SW_LOG_TABLE}, {BSG_SW_RSQRT_TABLE}, {BSG_SW_ANGLE_TABLE}, {BSG_SW_EXP2_TABLE}, \
     {BSG_SW_EXP_TABLE}}
