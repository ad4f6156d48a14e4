// bsg_fx64.h -- the double-precision price of one option (the formula and the
// final operations of price_fp64) with its elementary functions in 64-bit
// fixed point.
//
// Why: GB300 issues 2 double-precision operations per clock and SM; the
// formula takes 177 of them (four divisions, a square root, a log, three
// exps and two polynomials).  Here sqrt, log, exp and the division are integer
// work on the multiply-add pipes (as bsg_swmath.h, whose tables these share),
// the tail of N -- exp and polynomial together -- comes from a table of its
// Taylor coefficients (15 integer multiply-adds; 46 with exp, reciprocal and
// polynomial evaluated: 173 us), and six double operations are left: the
// products and the difference of the reference's last line, on N rounded to
// 2^-53 as the reference's 1 - (1 - N(|d|)) rounds it.
//
// 4M options: 1368 us in doubles, 122 us here.
//
// Precision (against long double, over max(s, k)): root mean square 6.0e-17
// and at most 3.2e-16 on strikes to 1.5 times the spot price, 1.1e-16 and
// 7.2e-16 in doubles; 5.7e-17 and 3.4e-16 on strikes to 20 times, 6.2e-17 and
// 5.4e-16 in doubles.  num = (r + v^2/2) t + ln(s/k), d1 and d2 carry 58 fraction bits
// (the double evaluation rounds ln(s/k) near 2^-53 and N to 2^-53), the
// tails of N 60; v sqrt(t) and 1/(v sqrt t) have 55 significant bits.
//
// Where the double evaluation is kept: one unit of N, 2^-53, is worth 2^-53 s
// or 2^-53 k e^(-rt), and for an option far out of the money that may be more
// of its price than the 1e-13 this mode is held to.  Which of two units a tail
// near the middle between them rounds to then is the double evaluation's own
// rounding error, so such an option (the middle within 4.5 (x^2 + 4) 2^-53 of
// the tail, the largest such error seen in 2M tails, and a unit worth more than
// 0.94e-13 (1 + price)) is left to price_fp64: 2 % of a book with strikes to 20
// times the spot price, none with strikes to 1.5 times.
//
// Domain (fx64_domain): every field's exponent and the products small enough
// that the fixed-point formats hold them -- v sqrt(t) in [2^-26, 4), |r t| <
// 4, s/k in 2^+-20, s and k in 2^+-80.
// Anything else (zeros, negative or enormous times, infinities, NaN) is
// priced by price_fp64 itself.
#pragma once
#include "bsg_fx64_tables.h"
#include "bsg_swmath.h"

namespace bsg_fx {

using bsg_sw::hi32;
using bsg_sw::hi32x32;
using bsg_sw::mul_64x32;
using bsg_sw::mulhi;
using bsg_sw::wide;

// Taylor coefficients of the upper tail on [i/64, (i + 1)/64): 64 fraction
// bits, then 59 (gen_fx64_tables.py).
struct alignas(16) TailEntry { uint64_t a0; int64_t a1, a2, a3; int32_t a4, a5, a6, a7; };
struct alignas(16) TailTable { TailEntry at[BSG_FX_TAIL_ENTRIES]; };  // 26,112 bytes

BSG_SW_FN int exponent_of(uint64_t b) { return (int)(b >> 52) & 2047; }
// The significand with its top bit at bit 63 (zero for a zero or denormal).
BSG_SW_FN uint64_t significand(uint64_t b) {
    return ((b & 0x7FF0000000000000ull) ? 0x8000000000000000ull : 0ull) | (b << 11 & 0x7FFFFFFFFFFFFFFFull);
}

BSG_SW_FN bool fx64_domain(uint64_t s, uint64_t k, uint64_t r, uint64_t v, uint64_t t) {
    const int es = (int)(s >> 52), ek = (int)(k >> 52), ev = (int)(v >> 52), et = (int)(t >> 52);
    const int er = exponent_of(r);  // of |r|
    // exponents with the sign bit: a negative field is out of range
    return (unsigned)(es - 943) <= 160u && (unsigned)(ek - 943) <= 160u && (unsigned)(es - ek + 20) <= 40u &&
           (unsigned)(ev - 983) <= 80u && (unsigned)(et - 983) <= 80u &&
           // v^2 t in [2^-52, 2^4), |r t| < 4
           (unsigned)(2 * ev + et - 3 * 1023 + 52) <= 53u && er + et - 2 * 1023 < 1;
}

// a + s e: s with 64 fraction bits, e with 32 (|e| <= 1/2); up to 3 units off.
BSG_SW_FN int64_t horner(int64_t a, int64_t s, int32_t e) {
    return a + (int64_t)(int32_t)(s >> 32) * e + (int64_t)bsg_sw::shi32x32((int32_t)((uint32_t)s >> 1), e) * 2;
}

// N's upper tail at x >= 0 (58 fraction bits) in units of 2^-53, rounded, from
// the table's Taylor polynomial of degree 7 (its error is under 2^-64).  Sets
// *near where the rounding is in doubt (above).
BSG_SW_FN uint64_t tail_units(const TailTable& t, uint64_t x, bool* near) {
    const uint64_t top = (17ull << 57) - 1;              // 8.5: from there on 0 units
    x = x < top ? x : top;
    const TailEntry& p = t.at[(int)(x >> 52)];
    const int32_t e = (int32_t)((uint32_t)(x >> 20) ^ 0x80000000u);   // 64 (x - middle), 32 bits
    int32_t h = p.a6 + bsg_sw::shi32x32(p.a7, e);
    h = p.a5 + bsg_sw::shi32x32(h, e);
    h = p.a4 + bsg_sw::shi32x32(h, e);
    const int64_t s3 = p.a3 + (int64_t)bsg_sw::shi32x32(h, e) * 32;
    const int64_t s2 = horner(p.a2, s3, e);
    const int64_t s1 = horner(p.a1, s2, e);
    // x's last 20 bits times the slope s1 + e (s2 + e s3)
    const int32_t slope = (int32_t)(s1 >> 32) +
        bsg_sw::shi32x32((int32_t)(s2 >> 32) + bsg_sw::shi32x32((int32_t)(s3 >> 32), e), e);
    const int32_t low = (int32_t)(((uint32_t)x & 0xFFFFFu) << 11);
    const uint64_t q = (uint64_t)(horner((int64_t)p.a0, s1, e) + (int64_t)bsg_sw::shi32x32(low, slope) * 2);  // 64
    // |q - middle| in 2^-11 units against 2^11 4.5 q (x^2 + 4), and this
    // evaluation's own 2^-60
    const uint32_t x16 = (uint32_t)(x >> 54), x2 = (x16 * x16) >> 8;
    const int d = (int)((uint32_t)q & 2047) - 1024;
    const uint32_t window = (((uint32_t)(q >> 40) * (x2 + 5) * 9) >> 14) + 12;
    *near = *near || (uint32_t)(d < 0 ? -d : d) < window;
    return (q + 1024) >> 11;
}

// A positive double (its bits) inside the floats' range as a float, truncated.
BSG_SW_FN float as_float(uint64_t b) {
    const uint32_t u = (uint32_t)((b - ((uint64_t)(1023 - 127) << 52)) >> 29);
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}
BSG_SW_FN float larger(float a, float b) { return a > b ? a : b; }

struct Seed2 { uint64_t root, rroot; int e; };

// sqrt and 1/sqrt of w = x 2^-s (x's top bit set): root 2^(e - 62) and
// rroot 2^(-e - 62).
template <typename Tables>
BSG_SW_FN Seed2 sqrt_both(const Tables& t, uint64_t x, int s) {
    const int b = 64 - s;
    const int odd = b & 1;
    const uint64_t y = x >> odd;
    uint32_t c;
    const uint32_t y0 = bsg_sw::rsqrt_seed(t, y, &c);
    const uint64_t s0 = mul_64x32(y, y0);
    return {s0 + (wide((uint32_t)(s0 >> 30), c) >> 26), ((uint64_t)y0 << 32) + (wide(y0, c) >> 24),
            (b + odd) / 2};
}

// The price for fields inside the domain (their bits), otype 0 = call; false
// where it is left to price_fp64.
template <typename Tables>  // bsg_sw::Tables, or one with its lg, rs and e2
BSG_SW_FN bool price_fx64(const Tables& t, const TailTable& tails, uint64_t bs, uint64_t bk, uint64_t br, uint64_t bv,
                          uint64_t bt, int otype, double* price) {
    const uint64_t ms = significand(bs), mk = significand(bk), mt = significand(bt), mv = significand(bv);
    const int es = exponent_of(bs), ek = exponent_of(bk), et = exponent_of(bt) - 1023, ev = exponent_of(bv) - 1023;
    // w = v^2 t, normalised
    uint64_t w = mulhi(mulhi(mv, mv), mt);               // (v^2 t) 2^(189 - 128 - 2 ev - et)
    const int nw = bsg_sw::clz64(w);                     // 0..2
    w <<= nw;
    const int sw = 61 + nw - 2 * ev - et;                // w 2^-sw
    const Seed2 den = sqrt_both(t, w, sw);
    // ln(s/k) = n ln 2 + (L(k) - L(s))/2
    int is, ik;
    int64_t r;
    const int64_t ls = bsg_sw::neg2_ln_core(t, ms, &is, &r), lk = bsg_sw::neg2_ln_core(t, mk, &ik, &r);
    const int n = es + (is >> 8) - ek - (ik >> 8);
    int64_t num = ((lk - ls) >> 5) + n * 0x02C5C85FDF473DE8ll;       // 58
    // r t
    const int er = exponent_of(br) - 1023;
    const uint64_t rt_m = mulhi(significand(br), mt);    // |r t| 2^(62 - er - et)
    const int rs = 4 - er - et;                          // >= 4
    const uint64_t rt = rs < 64 ? rt_m >> rs : 0;        // 58
    const bool rneg = (br >> 63) != 0;
    num += rneg ? -(int64_t)rt : (int64_t)rt;
    num += (int64_t)(w >> (sw - 57));                    // w/2: sw is 60 or more
    // d1 = num / (v sqrt t), d2 = d1 - v sqrt t, 58
    const bool dneg = num < 0;
    uint64_t an = dneg ? 0ull - (uint64_t)num : (uint64_t)num;
    an |= an == 0;
    const int nn = bsg_sw::clz64(an);
    const uint64_t dm = mulhi(an << nn, den.rroot);      // |d1| 2^(58 + nn + 62 - 64 + e)
    const int ds = nn + den.e - 2;
    const uint64_t far = 20ull << 58;                    // past every tail, and past 20 - 4 for d2
    uint64_t d1 = ds <= 0 ? far : ds < 64 ? dm >> ds : 0;
    d1 = d1 < far ? d1 : far;
    const uint64_t dd = den.root >> (4 - den.e);         // v sqrt t, 58
    const int64_t d2s = (dneg ? -(int64_t)d1 : (int64_t)d1) - (int64_t)dd;
    const bool d2neg = d2s < 0;
    bool near = false;
    const uint64_t q1 = tail_units(tails, d1, &near);
    const uint64_t q2 = tail_units(tails, d2neg ? 0ull - (uint64_t)d2s : (uint64_t)d2s, &near);
    // N(d1), N(d2) for a call, N(-d1), N(-d2) for a put, in units of 2^-53:
    // the tail where the sign says so, else 2^53 less the tail
    const bool put = otype != 0;
    const uint64_t s1 = dneg != put ? 0 : 1ull << 63, s2 = d2neg != put ? 0 : 1ull << 63;
    const double big = 4503599627370496.0;               // 2^52
    const double n1 = bsg_sw::add(bsg_sw::from_bits((0x4330000000000000ull + q1) ^ s1), s1 ? 3 * big : -big);
    const double n2 = bsg_sw::add(bsg_sw::from_bits((0x4330000000000000ull + q2) ^ s2), s2 ? 3 * big : -big);
    // k exp(-r t); both sides of the difference scaled by 2^-53
    const uint64_t xr = mulhi(rt, 0xB8AA3B295C17F0BCull);            // |r t| log2 e, 57
    const double ex = bsg_sw::exp2_fixed(t, rneg ? (int64_t)xr : -(int64_t)xr);
    const uint64_t down = 53ull << 52;
    const double fv = bsg_sw::mul(bsg_sw::from_bits(bk - down), ex);
    const double a = bsg_sw::mul(bsg_sw::from_bits(bs - down), n1), b = bsg_sw::mul(fv, n2);
    *price = put ? bsg_sw::add(b, -a) : bsg_sw::add(a, -b);
    // max(s, k e^(-rt)) against |price| as floats (the bits above a float's rounded off)
    const float worth = larger(as_float(bs), as_float(bsg_sw::to_bits(fv) + down));
    const uint64_t bp = bsg_sw::to_bits(*price) & 0x7FFFFFFFFFFFFFFFull;
    const float p = bp < (uint64_t)920 << 52 ? 0.0f : as_float(bp);
    return !(near && worth > 850.0f + 850.0f * p);
}

}  // namespace bsg_fx

// The table's initializer: `const bsg_fx::TailTable t = BSG_FX_TAILS;`
#define BSG_FX_TAILS {{BSG_FX_TAIL_TABLE}}
