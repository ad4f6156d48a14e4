"""The double price with its elementary functions in fixed point
(p3arsec_gb300/csrc/bsg_fx64.h): on the CPU, the host build of the same code
against the formula in long double and in double; on the GPU, the kernel at
the ends of the fixed-point domain against the double oracle."""
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "p3arsec_gb300", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fx64") / "fx64_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                    os.path.join(HERE, "fx64_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("dist,left_at_most", [(0, 0), (1, 0.03), (2, 1)], ids=["plain", "tails", "wide"])
def test_no_further_off_than_doubles(checker, dist, left_at_most):
    """Against long double, the fixed-point prices are no further off than the
    double evaluation (largest and root mean square; the largest with 1e-16 of
    room, a quarter of one rounding of N at s = k), and within the 1e-13 that
    the mode's tests hold it to of the double evaluation."""
    n = 300_000
    r = subprocess.run([checker, str(n), "11", str(dist)], stdout=subprocess.PIPE, text=True, check=True)
    m = re.match(r"priced (\d+) left (\d+) fixed (\S+) (\S+) double (\S+) (\S+) test (\S+)", r.stdout)
    priced, left = int(m[1]), int(m[2])
    f_max, f_rms, d_max, d_rms, test = (float(x) for x in m.groups()[2:])
    assert priced + left == n and left <= left_at_most * n and priced > n // 20, r.stdout
    assert f_max <= d_max + 1e-16 and f_rms <= d_rms, r.stdout
    if dist < 2:
        assert test <= 1.0, r.stdout


def test_table_header_is_what_the_generator_writes(tmp_path):
    """bsg_fx64_tables.h is generated: regenerating it changes nothing."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("gen_fx64", os.path.join(CSRC, "gen_fx64_tables.py"))
    gen = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(gen)
    gen.HERE = str(tmp_path)
    gen.main()
    with open(os.path.join(CSRC, "bsg_fx64_tables.h")) as a, open(tmp_path / "bsg_fx64_tables.h") as b:
        assert a.read() == b.read()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 255, 257, 152 * 3 * 256 + 1, 400_003])
def test_domain_ends_on_the_gpu(gpu_ctx, oracle_lib, n):
    """Books whose fields straddle the fixed-point domain (and its queue's
    room: over half of the options are left to the double evaluation), with
    zeros, infinities and NaN among them, through both FP64 entry points."""
    from p3arsec_gb300 import books
    rng = np.random.default_rng(n)
    book = books.generate(n, seed=n, dist="tails")
    s, k, r, v, t = (a.astype(np.float64) for a in book.arrays()[:5])
    wild = rng.random(n) < 0.6
    t[wild] = np.exp(rng.uniform(-20, 8, wild.sum()))
    v[wild] = np.exp(rng.uniform(-12, 3, wild.sum()))
    k[wild] = s[wild] * np.exp(rng.uniform(-20, 20, wild.sum()))
    for a, x in ((t, 0.0), (v, 0.0), (s, 0.0), (k, np.inf), (t, np.inf), (r, np.nan), (t, -1.0)):
        a[rng.random(n) < 0.01] = x
    arrays = [a.astype(np.float32) for a in (s, k, r, v, t)]
    wide = [a.astype(np.float64) for a in arrays]
    want = oracle_lib.price_fp64_d(*wide, book.otype)
    got, got32 = np.zeros(n), np.zeros(n)
    gpu_ctx.price_soa_f64(*wide, book.otype, got, num_runs=2)
    gpu_ctx.price_fp64(*arrays, book.otype, got32)
    assert np.array_equal(got.view(np.uint64), got32.view(np.uint64))
    # rtol, atol as the mode's other tests, scaled to strikes of up to e^20 s:
    # a unit of N is 2^-53 of the larger of s and k
    scale = np.maximum(np.maximum(wide[0], wide[1]), 1.0)
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~finite & ~np.isnan(want)], want[~finite & ~np.isnan(want)])
    off = np.abs(got[finite] - want[finite])
    assert np.all(off <= 1e-13 + 1e-13 * np.abs(want[finite]) + 2e-15 * scale[finite])
