// bsg_fx64.h -- the double-precision price of one option (the formula and the
// final operations of price_fp64) with its elementary functions in 64-bit
// fixed point.
//
// Why: GB300 issues 2 double-precision operations per clock and SM; the
// formula takes 177 of them (four divisions, a square root, a log, three
// exps and two polynomials).  Here sqrt, log, exp, the division and the
// polynomial are integer work on the multiply-add pipes (as bsg_swmath.h,
// whose tables these share), and six double operations are left: the
// products and the difference of the reference's last line, on N rounded to
// 2^-53 as the reference's 1 - (1 - N(|d|)) rounds it.
//
// 4M options: 1368 us in doubles, 175 us here.
//
// Precision (against long double, over max(s, k)): root mean square 6.0e-17
// and at most 3.2e-16 on strikes to 1.5 times the spot price, 1.1e-16 and
// 7.2e-16 in doubles; 5.7e-17 and 3.4e-16 on strikes to 20 times, 6.2e-17 and
// 5.4e-16 in doubles.  num = (r + v^2/2) t + ln(s/k), d1 and d2 carry 58 fraction bits
// (the double evaluation rounds ln(s/k) near 2^-53 and N to 2^-53), the
// tails of N 60; v sqrt(t) and 1/(v sqrt t) have 61 significant bits.
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
#include "bsg_swmath.h"

namespace bsg_fx {

using bsg_sw::hi32;
using bsg_sw::hi32x32;
using bsg_sw::mul_64x32;
using bsg_sw::mulhi;
using bsg_sw::wide;

#if defined(__CUDA_ARCH__)
// A reciprocal seed of y (62 fraction bits, [1, 4)) a few units of 2^-22 low:
// 1/y with 31 fraction bits.
BSG_SW_FN uint32_t rcp_seed(uint64_t y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_rn(hi32(y))));
    return __float2uint_rz(__fmul_rn(r, 2305841909702066176.0f));  // 2^61 (1 - 2^-21)
}
#else
inline uint32_t rcp_seed(uint64_t y) {
    return (uint32_t)((1.0f / (float)hi32(y)) * 2305841909702066176.0f);
}
#endif

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

// -2 ln of x = m 2^-63 in [1, 2) (for x >= 1.5 of x/2: *half = 1), 62 fraction bits.
BSG_SW_FN int64_t neg2_ln_significand(const bsg_sw::Tables& t, uint64_t m, int* half) {
    const int i = (int)((m >> 54) & 511);
    *half = i >> 8;
    const bsg_sw::LogEntry le = t.lg[i];
    const uint64_t lo = wide((uint32_t)m, le.c);
    const uint64_t hi = wide(hi32(m), le.c) + (lo >> 32);
    const int64_t r = (int64_t)((hi << 22) | ((uint32_t)lo >> 10));  // 73, as in neg2_ln_scaled
    const int32_t rh = (int32_t)(r >> 32);
    int32_t q = 858993459 - (bsg_sw::shi32x32(rh, 715827883) >> 9);
    q = 1073741824 - (bsg_sw::shi32x32(rh, q) >> 9);
    q = 1431655765 - (bsg_sw::shi32x32(rh, q) >> 9);
    const uint64_t q63 = (1ull << 63) - (uint64_t)(((int64_t)rh * q) >> 9);
    const uint64_t r2 = (uint64_t)((int64_t)rh * rh + 4) +
                        (uint64_t)((int64_t)bsg_sw::shi32x32(rh, (int32_t)((uint32_t)r >> 1)) * 4);
    return le.ln + (int64_t)(mulhi(r2, q63) >> 19) - (r >> 10);
}

// 2^(-x 2^-57) as a significand in [1, 2) (63 fraction bits) and *n >= 0, the
// power of two taken out; 0 < x 2^-57 < 63.
BSG_SW_FN uint64_t exp2_neg(const bsg_sw::Tables& t, uint64_t x, int* n) {
    const uint64_t f = 0ull - x;                                      // the fraction of -x
    const uint64_t a = (f & ((1ull << 47) - 1)) << 17;                // 74
    const uint64_t tt = mulhi(a, BSG_SW_LN2_64);
    const uint32_t th = hi32(tt);
    const uint64_t t2 = wide(th, th) + ((uint64_t)hi32x32(th, (uint32_t)tt) << 1);
    const uint32_t g = 2863311531u + hi32x32(th, 699051u);
    const uint64_t t3g = wide(hi32(t2), hi32x32(th, g));
    const uint64_t p = tt + (t2 >> 11) + (t3g >> 22);
    const uint64_t e = t.e2[(f >> 47) & 1023];
    *n = -(int)((int64_t)f >> 57);
    return e + (mulhi(e, p) >> 10);
}

// N's upper tail at x >= 0 (58 fraction bits) in units of 2^-53, rounded: the
// polynomial of Abramowitz and Stegun 26.2.17 with 1/sqrt(2 pi) multiplied
// into its coefficients.  Sets *near where the rounding is in doubt (above).
BSG_SW_FN uint64_t tail_units(const bsg_sw::Tables& t, uint64_t x, bool* near) {
    const uint64_t top = 2680624789467443200ull;         // 9.3: beyond it the tail is under 2^-66
    x = x < top ? x : top;
    // k = 1/(1 + c0 x): a seed 2^-21 low, then k0 (1 + e + e^2)
    const uint64_t y = (1ull << 62) + mulhi(x << 2, 0x3B4CE230E2201C00ull) * 4;  // 62
    const uint32_t k0 = rcp_seed(y);                     // 31
    const uint64_t e = (1ull << 61) - mul_64x32(y, k0);  // 61, in (0, 2^-20)
    const uint32_t eh = (uint32_t)(e >> 9);              // 52
    const uint64_t c = (e << 11) + hi32x32(eh, eh);      // e + e^2, 72
    const uint64_t k = ((uint64_t)k0 << 33) + (mul_64x32(c, k0) >> 7);  // 64
    const uint64_t a4 = 0xBA00E2B624772872ull - mulhi(k, 0x87DC2211AA9F6974ull);
    const uint64_t a3 = 0xB5F0E2AE93BD6878ull - mulhi(k, a4);
    const uint64_t a1 = 0x209E418D66AFA2E4ull + mulhi(k, mulhi(k, a3)) - mulhi(k, 0x246A6399C19DCB8Eull);
    const uint64_t p = mulhi(k, a1);                     // 64, at most 1/2
    // exp(-x^2/2) = 2^-(x^2 log2(e)/2); x in 60 bits, x^2 in 56
    const uint64_t xx = mulhi(x << 2, x << 2) << 1;
    int n;
    const uint64_t g = exp2_neg(t, mulhi(xx, 0xB8AA3B295C17F0BCull) | 1, &n);  // n >= 1
    const uint64_t q = mulhi(g, p) >> (n - 1);           // 64
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
BSG_SW_FN Seed2 sqrt_both(const bsg_sw::Tables& t, uint64_t x, int s) {
    const int b = 64 - s;
    const int odd = b & 1;
    const uint64_t y = x >> odd;
    const bsg_sw::SeedEntry se = t.rs[(int)(y >> 56) - 64];
    const uint32_t y0 = se.a - hi32x32(se.b, (uint32_t)(y >> 24));  // 30
    const uint64_t e = (1ull << 60) - mulhi(y, wide(y0, y0));
    const uint32_t eh = (uint32_t)(e >> 14);
    const uint32_t g = 805306368u + (hi32x32(eh, 671088640u) >> 14);
    const uint64_t corr = (e >> 1) + ((uint64_t)hi32x32(hi32(wide(eh, eh)), g) << 1);  // 60
    const uint64_t s0 = mul_64x32(y, y0);                            // 62
    return {s0 + (mulhi(s0, corr << 17) >> 13), ((uint64_t)y0 << 32) + (mul_64x32(corr << 17, y0) >> 13),
            (b + odd) / 2};
}

// The price for fields inside the domain (their bits), otype 0 = call; false
// where it is left to price_fp64.
BSG_SW_FN bool price_fx64(const bsg_sw::Tables& t, uint64_t bs, uint64_t bk, uint64_t br, uint64_t bv,
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
    int hs, hk;
    const int64_t ls = neg2_ln_significand(t, ms, &hs), lk = neg2_ln_significand(t, mk, &hk);
    const int n = es + hs - ek - hk;
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
    const uint64_t q1 = tail_units(t, d1, &near);
    const uint64_t q2 = tail_units(t, d2neg ? 0ull - (uint64_t)d2s : (uint64_t)d2s, &near);
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
