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
// of the cost.  Each series is cut where its terms pass 2^-60, and each term
// has the bits it needs for that and no more.  A normal variate, as a double,
// is within 1.5e-16 of max(1, |z|) of the exact one (5.0e-16 when every step was
// a double operation).
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
//  sqrt: a quadratic table seed at or below 1/sqrt(y) (384 intervals), then
//    s = y y0 (1 + e/2 + 3 e^2/8), e = 1 - y y0^2 < 2^-24 (the binomial series
//    of (1 - e)^(-1/2)).
//  sin/cos(2 pi u): the quadrant and the 1/2048 turn below u from k's bits,
//    the rest an exact integer; the angle-addition formulas combine the
//    table's sin and cos with Taylor polynomials of sin phi (to phi^5) and
//    cos phi (to phi^6), 0 < phi < 2 pi/2048: nothing is negative inside a
//    quadrant, so signs are set once, at the end.
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
struct alignas(16) SeedEntry { uint32_t a, b, c, unused; };
struct alignas(16) Angle { uint64_t s, c; };

// 31,232 bytes: the kernels copy it into shared memory once per block.
struct alignas(16) Tables {
    LogEntry lg[512];
    SeedEntry rs[384];  // y in [i/512, (i + 1)/512), i = 128..511
    Angle ang[512];     // the first quadrant
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

// -2 ln of x = m 2^-63 in [1, 2) with 62 fraction bits; for the upper half of
// the table (*i >= 256) that of x/2.  *r: x c - 1 (the table's c) with 63 bits.
template <typename T>
BSG_SW_FN int64_t neg2_ln_core(const T& t, uint64_t m, int* i, int64_t* r) {
    *i = (int)(m >> 54) & 511;
    const LogEntry le = t.lg[*i];
    // x c 2^83 = hi 2^32 + (lo mod 2^32); r = that less 2^83, exact before the shifts
    const uint64_t lo = wide((uint32_t)m, le.c);
    const uint64_t hi = wide(hi32(m), le.c) + (lo >> 32);
    *r = (int64_t)(((hi << 12) | ((uint32_t)lo >> 20)) ^ (1ull << 63));
    const int32_t rh = (int32_t)(uint32_t)(hi >> 10);    // r 2^41
    const int32_t nr = -(rh >> 9);                       // -r 2^32
    // -2 ln(1 + r) = -2 r + r^2 - r^2 r (2/3 - r (1/2 - r (2/5 - r/3)))
    int32_t q = 858993459 + shi32x32(nr, 715827883);     // 2/5 - r/3, 31 fraction bits
    q = 1073741824 + shi32x32(nr, q);
    q = 1431655765 + shi32x32(nr, q);
    const int32_t rq = (int32_t)(((int64_t)rh * q + (1ll << 30)) >> 31);  // 41
    const uint32_t rl = (uint32_t)((uint64_t)*r << 10);  // r 2^73 below rh's last bit
    // r^2 2^82, the cross term rounded down by at most 4: + 4 keeps it positive
    const uint64_t r2 = (uint64_t)((int64_t)rh * rh + 4) +
                        (uint64_t)((int64_t)shi32x32(rh, (int32_t)(rl >> 1)) * 4);
    uint32_t rs = (uint32_t)(r2 >> 31);                  // 51, below 2^31 but for |r| next to 2^-10
    rs = rs < 0x7FFFFFFFu ? rs : 0x7FFFFFFFu;
    const int64_t r3q = (int64_t)(int32_t)rs * rq;       // 51 + 41
    return le.ln + (int64_t)(r2 >> 20) - (r3q >> 30) - *r;
}

// -2 ln u for u = (2k + 1) 2^-53, k < 2^52, as x 2^-s with x's top bit set.
struct Scaled { uint64_t x; int s; };

BSG_SW_FN Scaled neg2_ln_scaled(const Tables& t, uint64_t k) {
    const uint64_t v = 2 * k + 1;                        // u = v 2^-53, v odd
    const int lz = clz64(v);                             // 11..63
    int i;
    int64_t r;
    const uint64_t w = (uint64_t)neg2_ln_core(t, v << lz, &i, &r);
    const int ne = lz - 10 - (i >> 8);                   // powers of two taken out, negated: 0..53
    if (ne == 0 && i == 511) {
        // u near 1: -2 ln u = 2 |r| (1 + c), c = |r|/2 + r^2/3 + |r|^3/4 + r^4/5,
        // |r| = 1 - u = (2^53 - v) 2^-53 with its top bit moved up
        const uint64_t ar = ((1ull << 53) - v) << 20;    // |r| 2^73
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
    // below 2 at ne = 0, where it may be small; below 73.5 otherwise
    const uint64_t x = ne == 0 ? w
                               : (uint64_t)((int64_t)w >> 5) + wide((uint32_t)BSG_SW_2LN2_57, (uint32_t)ne) +
                                     ((uint64_t)(hi32(BSG_SW_2LN2_57) * (uint32_t)ne) << 32);
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

// sqrt(w.x 2^-w.s) = s 2^(e - 62), s in [2^61, 2^62].
struct Root { uint64_t s; int e; };

// The seed and its correction: y (1/4..1, 64 fraction bits) -> y0 at or below
// 1/sqrt(y) (30) and c with 1/sqrt(y) = y0 (1 + c) (56).
template <typename T>
BSG_SW_FN uint32_t rsqrt_seed(const T& t, uint64_t y, uint32_t* c) {
    const SeedEntry se = t.rs[(int)(y >> 55) - 128];
    const uint32_t d = (uint32_t)(y >> 23);
    const uint32_t y0 = se.a - hi32x32(d, se.b - hi32x32(d, se.c));
    const uint64_t e = (1ull << 60) - mulhi(y, wide(y0, y0));        // 1 - y y0^2 in [0, 2^-24)
    const uint32_t h = (uint32_t)(e >> 5);               // e 2^55 = e/2 2^56
    *c = h + hi32x32(hi32x32(h, h), 384u);               // + 3 e^2/8: 78, 3/8 2^10, 56
    return y0;
}

BSG_SW_FN Root sqrt_scaled(const Tables& t, Scaled w) {
    const int b = 64 - w.s;                              // the value is (x 2^-64) 2^b
    const int odd = b & 1;
    const uint64_t y = w.x >> odd;                       // [1/4, 1), 64 fraction bits
    uint32_t c;
    const uint32_t y0 = rsqrt_seed(t, y, &c);
    const uint64_t s0 = mul_64x32(y, y0);                // 62, below 2^62
    return {s0 + (wide((uint32_t)(s0 >> 30), c) >> 26), (b + odd) / 2};
}

// 2 pi u (u = (2k + 1) 2^-53) less its whole quarter turns (k >> 50) as a
// table angle (63 fraction bits) and sin and cos (64) of the rest.
struct Turn { Angle a; uint64_t sn, cs; };

BSG_SW_FN Turn turn_of(const Tables& t, uint64_t k) {
    // phi = x 2 pi 2^-53, x = 2 (k mod 2^41) + 1: x 2^22 drops k's higher bits
    const uint64_t ph = mulhi((k << 23) | (1ull << 22), BSG_SW_2PI_53);  // 64
    const uint32_t phh = (uint32_t)(ph >> 24);           // 40
    const uint64_t p = wide(phh, phh) + ((uint64_t)hi32x32(phh, (uint32_t)ph << 8) << 1);  // phi^2, 80
    const uint32_t pp = hi32(p);                         // 48
    // sin = phi - phi phi^2 (1/6 - phi^2/120); the product with 58 bits
    const uint32_t sg = hi32x32(pp, 2863311531u - hi32x32(pp, 2185u));    // 34, 50
    const uint64_t sn = ph - ((uint64_t)hi32x32(phh, sg) << 6);           // 64
    // cos = 1 - phi^2/2 + phi^4 (1/24 - phi^2/720), less one unit: below 2^64
    const uint32_t f = hi32x32(pp, hi32x32(pp, 178956971u - hi32x32(pp, 91u)));  // 32, 48, 64
    return {t.ang[(int)(k >> 41) & 511], sn, f + ~(p >> 17)};
}

// sin and cos of the angle less its quarter turns, both >= 0, 63 bits.
BSG_SW_FN void sincos_quadrant(const Turn& r, uint64_t* s, uint64_t* c) {
    *s = mulhi(r.a.s, r.cs) + mulhi(r.a.c, r.sn);
    *c = mulhi(r.a.c, r.cs) - mulhi(r.a.s, r.sn);
}

// cos and sin of 2 pi u with 62 fraction bits.
BSG_SW_FN void sincos_2pi_fixed(const Tables& t, uint64_t k, int64_t* s, int64_t* c) {
    uint64_t s1, c1;
    sincos_quadrant(turn_of(t, k), &s1, &c1);
    const int q = (int)(k >> 50);
    const int64_t ss = (int64_t)(((q & 1) ? c1 : s1) >> 1), cc = (int64_t)(((q & 1) ? s1 : c1) >> 1);
    *s = (q & 2) ? -ss : ss;
    *c = ((q + 1) & 2) ? -cc : cc;
}

// A fixed-point value as a double.
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

// Normal variates with 58 fraction bits (|z| < 8.6) from four random words:
// u1 from (w0, w1), u2 from (w2, w3).  Negative ones are complemented, not
// negated: one unit of 2^-58 off.  With BOTH false *z1 is not computed.
constexpr int kZBits = 58;

template <bool BOTH>
BSG_SW_FN void normal_pair_fixed(const Tables& t, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3,
                                 int64_t* z0, int64_t* z1) {
    const Root r = sqrt_scaled(t, neg2_ln_scaled(t, unit_bits(w0, w1)));
    const Turn u = turn_of(t, unit_bits(w2, w3));
    const uint64_t r59 = (r.s << 1) >> (4 - r.e);        // e <= 4
    const bool odd = (w2 >> 30) & 1, upper = (w2 >> 31) & 1;
    const uint64_t m0 = 0ull - (uint64_t)(odd != upper), m1 = 0ull - (uint64_t)upper;
    uint64_t f0;                                         // |cos|: 59 + 63 - 64 bits times r
    if (BOTH) {
        uint64_t s, c;
        sincos_quadrant(u, &s, &c);
        f0 = odd ? s : c;
        *z1 = (int64_t)(mulhi(r59, odd ? c : s) ^ m1);
    } else {
        const uint64_t x = mulhi(odd ? u.a.s : u.a.c, u.cs), y = mulhi(odd ? u.a.c : u.a.s, u.sn);
        f0 = odd ? x + y : x - y;
    }
    *z0 = (int64_t)(mulhi(r59, f0) ^ m0);
}

// The same as doubles.
BSG_SW_FN void normal_pair(const Tables& t, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3,
                           double* z0, double* z1) {
    int64_t a, b;
    normal_pair_fixed<true>(t, w0, w1, w2, w3, &a, &b);
    *z0 = fixed_to_double(a, kZBits);
    *z1 = fixed_to_double(b, kZBits);
}

// 2^(f 2^-57) for the fraction of f 2^-57 alone: [1, 2), 63 fraction bits.
template <typename T>
BSG_SW_FN uint64_t exp2_fraction(const T& t, uint64_t f) {
    const uint64_t tt = mulhi(f << 17, BSG_SW_LN2_54);   // t = r ln 2, r < 2^-10 (74 bits): 64
    const uint32_t th = (uint32_t)(tt >> 22);            // 42
    const uint64_t t2 = wide(th, th) + ((uint64_t)hi32x32(th, (uint32_t)tt << 10) << 1);  // t^2, 84
    // t^3 (1/6 + t/24): 34, 44, then 52 + 44 - 32 = 64
    const uint32_t t3 = hi32x32(hi32(t2), hi32x32(th, 2863311531u + hi32x32(th, 699051u)));
    const uint64_t e = t.e2[(int)(f >> 47) & 1023];
    return e + mulhi(e, tt + (t2 >> 21) + t3);
}

// 2^(x 2^-57), |x 2^-57| < 64, as a double.
constexpr int kXBits = 57;
template <typename T>
BSG_SW_FN double exp2_fixed(const T& t, int64_t x) {
    const uint64_t y = exp2_fraction(t, (uint64_t)x);
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
