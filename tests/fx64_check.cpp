// CPU check of the fixed-point double price (p3arsec_gb300/csrc/bsg_fx64.h,
// the same code the GPU runs) against the formula in long double and in double.
//
//   fx64_check <n> <seed> <dist>     dist: 0 plain, 1 tails, 2 wide
// prints "priced <a> left <b> fixed <max> <rms> double <max> <rms> test <d>":
// errors over max(s, k), for the options priced in fixed point; d: the
// largest |fixed - double| / (1e-13 + 1e-13 |double|).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "bsg_fx64.h"

namespace {

const bsg_sw::Tables kT = BSG_SW_TABLES;
const bsg_fx::TailTable kTails = BSG_FX_TAILS;

template <typename F>
F upper_tail(F x) {  // the reference's polynomial, blackscholes.simd.c:134-216
    const F np = std::exp(F(-0.5) * x * x) * F(0.39894228040143270286);
    const F k = F(1) / (F(1) + F(0.2316419) * x);
    const F k2 = k * k, k3 = k2 * k, k4 = k3 * k, k5 = k4 * k;
    F l2 = k2 * F(-0.356563782) + k3 * F(1.781477937);
    l2 = l2 + k4 * F(-1.821255978);
    l2 = l2 + k5 * F(1.330274429);
    return (l2 + k * F(0.319381530)) * np;
}

template <typename F>
F cndf(F x) {
    const F out = F(1) - upper_tail(x < 0 ? -x : x);
    return x < 0 ? F(1) - out : out;
}

// long double: N is rounded to 64 bits, far below a double's unit
template <typename F>
F price(double s, double k, double r, double v, double t, int put) {
    const F den = F(v) * std::sqrt(F(t));
    const F d1 = ((F(r) + F(v) * F(v) * F(0.5)) * F(t) + std::log(F(s) / F(k))) / den, d2 = d1 - den;
    const F n1 = cndf(d1), n2 = cndf(d2), fv = F(k) * std::exp(-F(r) * F(t));
    return put ? fv * (F(1) - n2) - F(s) * (F(1) - n1) : F(s) * n1 - fv * n2;
}

uint64_t state;
double unit() {  // splitmix64
    uint64_t z = (state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (double)((z ^ (z >> 31)) >> 11) * 0x1.0p-53;
}

}  // namespace

int main(int argc, char** argv) {
    if (argc != 4) return 2;
    const long n = atol(argv[1]);
    state = strtoull(argv[2], nullptr, 10);
    const int dist = atoi(argv[3]);
    long priced = 0, left = 0;
    double mf = 0, md = 0, sf = 0, sd = 0, test = 0;
    for (long i = 0; i < n; ++i) {
        double s = 10 + 190 * unit(), k, t, r = 0.01 + 0.09 * unit(), v = 0.05 + 0.6 * unit();
        const int put = unit() < 0.5;
        if (dist == 0) {
            k = s * (0.5 + unit());
            t = 0.05 + 1.95 * unit();
        } else if (dist == 1) {
            k = s * (0.05 + 19.95 * unit());
            t = 0.001 + 4.999 * unit();
        } else {  // past the domain's ends on every side
            s = std::exp(120 * unit() - 60);
            k = s * std::exp(30 * unit() - 15);
            t = std::exp(34 * unit() - 30);
            v = std::exp(24 * unit() - 20);
            r = (unit() - 0.4) * std::exp(12 * unit() - 10);
        }
        if (i & 1) {
            s = (float)s, k = (float)k, t = (float)t, r = (float)r, v = (float)v;
        }
        const uint64_t b[5] = {bsg_sw::to_bits(s), bsg_sw::to_bits(k), bsg_sw::to_bits(r),
                               bsg_sw::to_bits(v), bsg_sw::to_bits(t)};
        double f;
        if (!bsg_fx::fx64_domain(b[0], b[1], b[2], b[3], b[4]) ||
            !bsg_fx::price_fx64(kT, kTails, b[0], b[1], b[2], b[3], b[4], put, &f)) {
            ++left;
            continue;
        }
        ++priced;
        const double d = price<double>(s, k, r, v, t, put);
        const long double x = price<long double>(s, k, r, v, t, put);
        const double scale = s > k ? s : k;
        const double ef = std::fabs((double)(f - x)) / scale, ed = std::fabs((double)(d - x)) / scale;
        mf = std::fmax(mf, ef), md = std::fmax(md, ed), sf += ef * ef, sd += ed * ed;
        test = std::fmax(test, std::fabs(f - d) / (1e-13 + 1e-13 * std::fabs(d)));
    }
    printf("priced %ld left %ld fixed %.4e %.4e double %.4e %.4e test %.4f\n", priced, left, mf,
           std::sqrt(sf / priced), md, std::sqrt(sd / priced), test);
    return 0;
}
