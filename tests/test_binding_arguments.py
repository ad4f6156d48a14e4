"""What the binding's native half takes as an argument, without a GPU: the calls
go to no context (status -1), so an argument that is refused raises before."""
import ctypes
import dataclasses
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from p3arsec_gb300 import abi, build
from p3arsec_gb300 import swaptions as S

INVALID = -1


@pytest.fixture(scope="module")
def call():
    build.build()
    abi.load()
    return abi._call


def _host(n):
    return [np.ones(n, np.float32) for _ in range(5)] + [np.zeros(n, np.int32), np.zeros(n, np.float32)]


COUNTS = {"float": 100.0, "fraction": 2.5, "text": "100", "bytes": b"100", "numpy float": np.float64(2)}
TAKEN = {"int": 3, "bool": True, "numpy int": np.int64(3), "numpy unsigned": np.uint8(3)}


def _calls(call):
    """Every count of every call, as a function of its value."""
    host, sw = _host(100), S.generate(1, 1)
    one = np.zeros(1)
    price = lambda n=1, runs=1, flags=0: call.price_soa(0, *host, n, runs, flags, False)  # noqa: E731
    batch = lambda n=1, runs=1, flags=1: call.price_batch(0, (0,) * 6, 0, n, [(0, 1)], runs, flags, False)  # noqa: E731
    return {
        "n": lambda x: price(n=x), "num_runs": lambda x: price(runs=x), "flags": lambda x: price(flags=x),
        "pool_len": lambda x: batch(n=x), "batch num_runs": lambda x: batch(runs=x),
        "batch flags": lambda x: batch(flags=x),
        "request n": lambda x: call.server_submit(0, *[a.ctypes.data for a in host], x)[0],
        "request id": lambda x: call.server_wait(0, x, 0.0)[0],
        "trials": lambda x: call.price_swaptions(0, tuple(sw), x, one, one),
        "seed": lambda x: call.price_swaptions(0, (dataclasses.replace(sw[0], seed=x),), 2, one, one),
    }


@pytest.mark.parametrize("value", list(COUNTS.values()), ids=list(COUNTS))
def test_counts_that_are_not_whole_are_refused(call, value):
    with pytest.raises(TypeError):
        ctypes.c_size_t(value)  # as ctypes refuses them
    for name, f in _calls(call).items():
        with pytest.raises(TypeError):
            print(name, f(value))


@pytest.mark.parametrize("value", list(TAKEN.values()), ids=list(TAKEN))
def test_whole_counts_are_taken(call, value):
    for name, f in _calls(call).items():
        assert f(value) == INVALID, name


def test_segments_take_what_int_takes(call):
    batch = lambda segs: call.price_batch(0, (0,) * 6, 0, 100, segs, 1, 1, False)  # noqa: E731
    for segs in ([(0, 5)], [(0.0, 5.5)], [("0", "5")], [[0, 5]], np.array([[0, 5], [7, 2]]), (), [(np.int32(0), 2)]):
        assert batch(segs) == INVALID
    for segs, e in (([(0,)], ValueError), ([(0, 1, 2)], ValueError), ([(0, "x")], ValueError), ([(0, None)], TypeError),
                    ([5], TypeError), (5, TypeError)):
        with pytest.raises(e):
            batch(segs)


def test_host_arrays_at_any_address(call):
    """Arrays of the right type that begin at an odd address (a field of a packed
    record, a view of a file's bytes) are taken; the other byte order is not."""
    for off in (1, 2, 3):
        odd = [np.zeros(44, np.uint8)[off:off + 40].view(a.dtype) for a in _host(10)]
        assert not odd[0].flags.aligned
        assert call.price_soa(0, *odd, 10, 1, 0, False) == INVALID
        for i in range(7):
            swapped = list(odd)
            swapped[i] = odd[i].view(odd[i].dtype.newbyteorder())
            with pytest.raises(TypeError):
                call.price_soa(0, *swapped, 10, 1, 0, False)


MEMORY = r"""
import resource, sys
from p3arsec_gb300 import abi, swaptions
abi.load()
kind = sys.argv[1]
if kind == "segments":
    items = [(0, 1)] * (1 << 24)   # 128 MB here, 256 MB as segments
    call = lambda: abi._call.price_batch(0, (0,) * 6, 0, 100, items, 1, 1, False)
else:
    items = tuple(swaptions.generate(1, 1)) * (1 << 22)  # 32 MB here, 400 MB as structs
    call = lambda: abi._call.price_swaptions(0, items, 2, 0, 0)
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (128 << 20),) * 2)
try:
    call()
except MemoryError:
    print("refused")
"""


@pytest.mark.parametrize("kind", ["segments", "swaptions"])
def test_no_memory_is_an_exception(call, kind):
    """In a process with too little address space for the call's own table."""
    r = subprocess.run([sys.executable, "-c", MEMORY, kind], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT),
                       stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "refused", (r.returncode, r.stderr[-500:])


def test_items_that_change_the_callers_list(call):
    """Reading a segment or a swaption may run Python code; what the call reads is
    what the list held when it was given."""
    segs = []

    class Clears:
        def __init__(self, x):
            self.x = x

        def __int__(self):
            segs.clear()
            return self.x

    for pair in (lambda o: (Clears(o), 1), lambda o: [Clears(o), 1]):
        segs[:] = [(0, 1)] * 100 + [pair(500 + i) for i in range(1000)]
        assert call.price_batch(0, (0,) * 6, 0, 2000, segs, 1, 1, False) == INVALID
        assert segs == []
    mine = []

    @dataclasses.dataclass
    class Shrinks(S.Swaption):
        @property
        def n_steps(self):
            mine.clear()
            return 11

    class NoGpu(abi.Context):
        def __init__(self):
            self.lib, self.h, self._addr = abi.load(), None, None

    mine[:] = [Shrinks(strike=0.1, years=5.5, seed=i) for i in range(500)]
    with pytest.raises(abi.BsgError):
        NoGpu().price_swaptions(mine, 2)
    assert mine == []
