"""A program that has asked the driver to block while it waits (the device's
schedule flags) is not made to spin by the calls that poll their kernel's word.
In a process of its own: the flags belong to the device's primary context."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes, sys, time
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
assert cu.cuDevicePrimaryCtxSetFlags_v2(0, int(sys.argv[1])) == 0
import numpy as np, torch
from p3arsec_gb300 import Context, books
n, runs = 1 << 22, 10  # about 1.2 ms, below the polling's limit
book = books.generate(n, seed=3)
cols = [torch.from_numpy(a).cuda() for a in book.arrays()]
cols = [c.double() for c in cols[:5]] + [cols[5], torch.zeros(n, dtype=torch.float64, device="cuda:0")]
torch.cuda.synchronize()
with Context(0, 1) as ctx:
    call = lambda: ctx.price_soa_f64(*cols, n=n, num_runs=runs, device=True)
    for _ in range(10):
        call()
    w, c = time.perf_counter(), time.thread_time()
    for _ in range(200):
        call()
    w, c = time.perf_counter() - w, time.thread_time() - c
print(w, c)
"""


@pytest.mark.parametrize("flags,lo,hi", [(0x04, 0.0, 0.5), (0x01, 0.5, 1.1)], ids=["block", "spin"])
def test_schedule_flags_hold(flags, lo, hi):
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(flags)], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT),
                       stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    wall, cpu = (float(x) for x in r.stdout.split()[-2:])
    assert lo < cpu / wall < hi, (wall, cpu)
