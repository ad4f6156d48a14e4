"""Writes bsg_fx64_tables.h: the table of the CNDF's upper tail in bsg_fx64.h.

The function is the reference's, q(x) = exp(-x^2/2)/sqrt(2 pi) P(1/(1 + c0 x))
with the polynomial of Abramowitz and Stegun 26.2.17, its constants the
doubles the reference's literals are.  Entry i holds the Taylor coefficients
of q at the middle of [i/64, (i + 1)/64) in the variable e = 64 (x - middle),
|e| <= 1/2, from exact series arithmetic with 60 digits: 64 fraction bits for
the first four, 59 for the next four.

    python gen_fx64_tables.py      # rewrites bsg_fx64_tables.h here"""
import decimal
import os

decimal.getcontext().prec = 60
D = decimal.Decimal
HERE = os.path.dirname(os.path.abspath(__file__))
ENTRIES = 544  # x < 8.5: q(8.5) is a tenth of 2^-53
N = 8          # coefficients
C0 = D(0.2316419)
C = [D(0.319381530), D(-0.356563782), D(1.781477937), D(-1.821255978), D(1.330274429)]
INV_SQRT_2PI = D(0.39894228040143270286)


def mul(a, b):
    out = [D(0)] * N
    for i, x in enumerate(a):
        for j, y in enumerate(b[:N - i]):
            out[i + j] += x * y
    return out


def tail_series(x0):
    """Taylor coefficients of q at x0 in x - x0."""
    k0 = 1 / (1 + C0 * x0)
    k = [k0 * (-C0 * k0) ** n for n in range(N)]
    p = [D(0)] * N
    for c in reversed(C):  # Horner over series: p = k (c + p)
        p[0] += c
        p = mul(p, k)
    # exp(-(x0 d + d^2/2)): e' = -(x0 + d) e
    e = [D(1)] + [D(0)] * (N - 1)
    for n in range(1, N):
        e[n] = -(x0 * e[n - 1] + (e[n - 2] if n > 1 else D(0))) / n
    g = (-x0 * x0 / 2).exp() * INV_SQRT_2PI
    return [g * v for v in mul(p, e)]


def fixed(v, bits):
    return int((v * D(2) ** bits).to_integral_value(decimal.ROUND_HALF_EVEN))


def main():
    out = ["// bsg_fx64_tables.h -- written by gen_fx64_tables.py; do not edit.",
           "// The CNDF's upper tail by its Taylor coefficients on 1/64 intervals.",
           "#pragma once", "", f"#define BSG_FX_TAIL_ENTRIES {ENTRIES}", "#define BSG_FX_TAIL_TABLE \\"]
    for i in range(ENTRIES):
        a = [v / D(64) ** n for n, v in enumerate(tail_series((D(i) + D("0.5")) / 64))]
        w = [f"{fixed(a[0], 64)}ull"] + [f"{fixed(v, 64)}ll" for v in a[1:4]] + [f"{fixed(v, 59)}" for v in a[4:]]
        assert all(abs(fixed(v, 59)) < 2 ** 31 for v in a[4:])
        out.append("    {" + ", ".join(w) + "}" + (", \\" if i < ENTRIES - 1 else ""))
    with open(os.path.join(HERE, "bsg_fx64_tables.h"), "w") as f:
        f.write("\n".join(out) + "\n")


if __name__ == "__main__":
    main()
