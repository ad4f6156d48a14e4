"""The swaption kernel's exponents on the GPU against the CPU oracle
(oracle/swpt_oracle.c) on the same paths: every number of them at which the
kernel takes another body (1-4, 5-8, more, none that pays), both with and
without a path-dependent discount, and rates outside the fixed-point range,
which the kernel evaluates in double precision.

Tolerances as in test_gpu_swaptions.py (price relative 1e-10, absolute 1e-12;
standard error relative 1e-6): both sides evaluate exponents of magnitude X
to about X 2^-53 relative, 1e-14 at the largest here (X < 100)."""
import numpy as np
import pytest

from p3arsec_gb300 import swaptions as S

pytestmark = pytest.mark.gpu


def _sw(n, h, maturity, tenor, pay, strike=0.05, vol=0.01, nf=3, seed=11):
    rng = np.random.default_rng(seed)
    return S.Swaption(strike=strike, years=n * h, maturity=maturity * h, tenor=tenor * h,
                      payment_interval=pay * h, yield_curve=0.03 + 0.001 * np.arange(n),
                      factors=rng.uniform(-0.3 * vol, vol, (nf, n - 1)), seed=seed)


CASES = {
    "one": _sw(11, 1.0, 1, 1, 1),
    "one_and_discount": _sw(11, 1.0, 2, 1, 1, nf=1),
    "three": _sw(12, 0.5, 1, 3, 1),
    "four": _sw(12, 0.5, 3, 3, 1, nf=2),
    "five": _sw(12, 0.5, 1, 5, 1),
    "eight": _sw(20, 0.25, 2, 7, 1, nf=5),
    "nine": _sw(20, 0.25, 2, 8, 1),
    "thirty": _sw(32, 0.25, 1, 30, 1),
    "most_coefficients": _sw(32, 0.25, 16, 15, 1, nf=8, vol=0.004),
    "none_pays": _sw(11, 1.0, 1, 2, 3),
    "no_last_payment": _sw(11, 0.5, 2, 5, 2),
    "zero_strike": _sw(11, 1.0, 1, 2, 1, strike=0.0),
    "wide_coefficients": _sw(20, 1.0, 2, 10, 1, vol=0.12),
    "wide_constant": _sw(32, 1.0, 1, 30, 2, vol=0.08, strike=1.5),
}


@pytest.mark.parametrize("trials", [2, 257, 20_001])
def test_every_number_of_exponents(gpu_ctx, oracle_lib, trials):
    sw = list(CASES.values())
    got, err = gpu_ctx.price_swaptions(sw, trials)
    for (name, w), p, e in zip(CASES.items(), got, err):
        want, want_err = oracle_lib.swaption_price(w, trials)
        assert p == pytest.approx(want, rel=1e-10, abs=1e-12), name
        assert e == pytest.approx(want_err, rel=1e-6, abs=1e-14, nan_ok=True), name


def test_alone_and_among_others(gpu_ctx):
    """One launch's shape for small tables and one for large: the same bits."""
    got, err = gpu_ctx.price_swaptions(list(CASES.values()) * 5, 30_000)
    for i, w in enumerate(CASES.values()):
        p, e = gpu_ctx.price_swaptions([w], 30_000)
        assert p[0].tobytes() == got[i].tobytes() and e[0].tobytes() == err[i].tobytes()
