"""The libm mode's own division, square root and reciprocal (two at a time)
against CUDA's correctly rounded ones, bit for bit: every argument that the mode
can give the latter two, and 2^36 pairs of operands of the first, random, next
to powers of two, and with quotients next to the middle of two floats.  (A wrong
rounding of one in 2^30 quotients would go unseen by any book of options.)"""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT
from p3arsec_gb300 import build as b


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("rounding") / "librounding.so")
    r = subprocess.run([b.nvcc()] + b.NVCC_FLAGS + ["-shared", os.path.join(ROOT, "tests", "rounding_check.cu"),
                                                    "-o", so], stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                       text=True)
    assert r.returncode == 0, r.stdout
    L = ctypes.CDLL(so)
    for f in (L.check_unary, L.check_div):
        f.restype = ctypes.c_longlong
    L.check_unary.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p]
    L.check_div.argtypes = [ctypes.c_ulonglong, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return L


def test_the_check_compiles(lib):
    assert lib.check_div


@pytest.mark.gpu
@pytest.mark.parametrize("sqrt,lo,hi", [(0, -60, 110), (1, -40, 40)], ids=["reciprocal", "square root"])
def test_every_argument(lib, sqrt, lo, hi):
    bad = ctypes.c_ulonglong()
    n = lib.check_unary(sqrt, lo, hi, ctypes.byref(bad))
    assert n == 0, (n, hex(bad.value))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,launches", [(0, 32), (1, 4), (2, 28)], ids=["random", "powers of two", "midpoints"])
def test_quotients(lib, kind, launches):
    bad = ctypes.c_ulonglong()
    n = lib.check_div(7, launches, kind, ctypes.byref(bad))
    assert n == 0, (n, hex(bad.value))
