"""Writes bsg_swmath_tables.h: the tables of the fixed-point Box-Muller
transform and power of two and of the double-precision exponential in
bsg_swmath.h, computed from 70-digit decimal values of ln 2, ln c, sin, cos,
1/sqrt(y), 2^(j/1024) and 2^(j/64) and rounded once.

    python gen_swmath_tables.py      # rewrites bsg_swmath_tables.h here

Doubles are written as hex literals and fixed-point values as integers, so
the header is exact."""
import decimal
import os
from fractions import Fraction

decimal.getcontext().prec = 70
D = decimal.Decimal
HERE = os.path.dirname(os.path.abspath(__file__))


def round_bits(v: Fraction, bits: int) -> Fraction:
    """v rounded to `bits` significant bits, ties to even."""
    if v == 0:
        return Fraction(0)
    a = abs(v)
    e = a.numerator.bit_length() - a.denominator.bit_length()
    if Fraction(2) ** e > a:
        e -= 1
    scale = Fraction(2) ** (bits - 1 - e)
    return round(v * scale) / scale


def f64(v) -> float:
    x = round_bits(Fraction(v), 53)
    d = float(x)
    assert Fraction(d) == x, "not representable"
    return d


def hexd(v) -> str:
    d = f64(v)
    return d.hex() if d != 0 else "0.0"


def fixed(v, bits: int) -> int:
    """v with `bits` fraction bits, rounded to nearest."""
    return round(Fraction(v) * 2 ** bits)


def hexu(v, bits: int) -> str:
    x = fixed(v, bits)
    assert 0 <= x < 1 << 64
    return f"0x{x:016X}ull"


def atan_inv(x: int) -> D:
    """atan(1/x) by its Taylor series."""
    s, term, k, x2 = D(0), D(1) / D(x), 0, D(x) * D(x)
    while abs(term) > D(10) ** -75:
        s += term / (2 * k + 1) if k % 2 == 0 else -term / (2 * k + 1)
        term /= x2
        k += 1
    return s


PI = 16 * atan_inv(5) - 4 * atan_inv(239)  # Machin's formula


def sin_cos(x: D):
    """sin x and cos x by their Taylor series (|x| <= 2 pi)."""
    s, c = D(0), D(0)
    term, n = D(1), 0  # term = x^n / n!
    while n < 200:
        if n % 4 == 0:
            c += term
        elif n % 4 == 1:
            s += term
        elif n % 4 == 2:
            c -= term
        else:
            s -= term
        n += 1
        term = term * x / n
        if n > 10 and abs(term) < D(10) ** -75:
            break
    tiny = D(10) ** -60  # the zeros of sin and cos at multiples of pi / 2
    return (D(0) if abs(s) < tiny else s), (D(0) if abs(c) < tiny else c)


def main():
    ln2 = D(2).ln()
    out = []
    w = out.append
    w("// bsg_swmath_tables.h -- written by gen_swmath_tables.py; do not edit.")
    w("// Tables of the fixed-point Box-Muller transform, 2^x and exp in bsg_swmath.h.")
    w("#pragma once")
    w("")
    w("// fixed-point constants: 2 ln 2 (57 fraction bits), 2 pi (53), ln 2 (54)")
    w(f"#define BSG_SW_2LN2_57 {hexu(2 * ln2, 57)}")
    w(f"#define BSG_SW_2PI_53 {hexu(2 * PI, 53)}")
    w(f"#define BSG_SW_LN2_54 {hexu(ln2, 54)}")
    w("")
    w("// {2 ln c (62 fraction bits), c (20)}, c the reciprocal of the middle of")
    w("// interval i of [1, 2), i = 0..511; 2 ln(2 c) from i = 256 on; c = 1/2 for the last")
    w("#define BSG_SW_LOG_TABLE \\")
    for i in range(512):
        c = 2 ** 19 if i == 511 else round(Fraction(2 ** 20) * Fraction(1024, 1024 + 2 * i + 1))
        v = 2 * (D(c) / D(2) ** 20 * (2 if i >= 256 else 1)).ln()
        w(f"    {{{fixed(v, 62)}ll, {c}u}}" + (", \\" if i < 511 else ""))
    w("")
    w("// {a, b, c} (30 fraction bits), i = 128..511: a - d (b - c d) is at or")
    w("// below 1/sqrt(y) for y = (i + d)/512, d in [0, 1)")
    w("#define BSG_SW_RSQRT_TABLE \\")
    for i in range(128, 512):
        # the parabola through the curve at the three Chebyshev points, moved
        # down by its largest error (three 30-bit units for the roundings)
        y0, h = D(i) / 512, D(1) / 512
        f = lambda d: 1 / (y0 + h * d).sqrt()  # noqa: E731
        c3 = D(3).sqrt() / 4
        x = [D("0.5") - c3, D("0.5"), D("0.5") + c3]
        f0, f1, f2 = (f(v) for v in x)
        d01, d12 = (f1 - f0) / (x[1] - x[0]), (f2 - f1) / (x[2] - x[1])
        q = (d12 - d01) / (x[2] - x[0])
        lin = d01 - q * (x[0] + x[1])
        con = f0 - x[0] * d01 + q * x[0] * x[1]
        over = max(con + lin * D(k) / 64 + q * (D(k) / 64) ** 2 - f(D(k) / 64) for k in range(65))
        a = int((con - over) * 2 ** 30) - 3
        w(f"    {{{a}u, {fixed(-lin, 30)}u, {fixed(q, 30)}u, 0u}}" + (", \\" if i < 511 else ""))
    w("")
    w("// {sin, cos}(2 pi j / 2048) (63 fraction bits), j = 0..511")
    w("#define BSG_SW_ANGLE_TABLE \\")
    for j in range(512):
        sj, cj = sin_cos(2 * PI * D(j) / D(2048))
        w(f"    {{{hexu(sj, 63)}, {hexu(cj, 63)}}}" + (", \\" if j < 511 else ""))
    w("")
    w("// 2^(j/1024) (63 fraction bits), j = 0..1023")
    w("#define BSG_SW_EXP2_TABLE \\")
    for j in range(1024):
        w(f"    {hexu((D(j) / D(1024) * ln2).exp(), 63)}" + (", \\" if j < 1023 else ""))
    w("")
    w("// exp: 64/ln 2, and ln2/64 = L1 + L2")
    L = ln2 / 64
    L1 = f64(L)
    w(f"#define BSG_SW_INV_L {hexd(1 / L)}")
    w(f"#define BSG_SW_L1 {hexd(L)}")
    w(f"#define BSG_SW_L2 {hexd(Fraction(L) - Fraction(L1))}")
    w("")
    w("// 2^(j/64), j = 0..63")
    w("#define BSG_SW_EXP_TABLE \\")
    for j in range(64):
        w(f"    {hexd((D(j) / D(64) * ln2).exp())}" + (", \\" if j < 63 else ""))
    w("")
    with open(os.path.join(HERE, "bsg_swmath_tables.h"), "w") as f:
        f.write("\n".join(out) + "\n")


if __name__ == "__main__":
    main()
