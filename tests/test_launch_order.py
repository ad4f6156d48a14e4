"""Calls on one context are ordered: a call's first pass waits for everything
that the stream holds, also where its passes are launched one by one
(BSG_NO_GRAPH) and programmatically.  On the CPU the launch attribute of every
shape's passes; on the GPU chains of asynchronous calls, each the next one's
input, against the same calls with a synchronisation between."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from p3arsec_gb300 import Context, books
from p3arsec_gb300 import build as b

N = 4_000_037  # a persistent grid and a resident prefix where untuned
SHAPES = [None, (1, 128, 0, 2, 1), (1, 128, 4, 7, 1, 10), (1, 256, 2, 2, 1), (1, 256, 0, 4, 1)]


def test_first_pass_is_never_programmatic(tmp_path):
    exe = str(tmp_path / "order")
    r = subprocess.run([b.nvcc(), "-std=c++17", "-I" + b.CSRC, "-I" + os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "launch_order_check.cpp"), "-o", exe],
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout


def _book(torch, n, seed):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in books.generate(n, seed=seed).arrays()]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_a_call_reads_what_the_call_before_it_wrote(shape):
    torch = pytest.importorskip("torch")
    s, k, r, v, t, o = _book(torch, N, 31)
    k = k.abs() + 1.0
    outs = [[torch.zeros(N, device="cuda:0") for _ in range(4)] for _ in range(2)]
    torch.cuda.synchronize()
    with Context(0, 1) as ctx:
        if shape:
            ctx.set_tune(*shape)
        for wait, (a, x, y, z) in zip((True, False), outs):
            # a graph or one pass, then passes launched one by one, each call's
            # prices the next one's strikes
            for runs, graph, strikes, out in ((1, True, k, a), (2, False, a, x), (3, False, x, y), (2, True, y, z)):
                ctx.price_soa(s, strikes, r, v, t, o, out, n=N, num_runs=runs, device=True, asynchronous=True,
                              graph=graph)
                if wait:
                    ctx.synchronize()
            ctx.synchronize()
    for one, two in zip(*outs):
        assert torch.equal(one.view(torch.int32), two.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_the_last_of_two_calls_with_one_price_array_stays(shape):
    torch = pytest.importorskip("torch")
    first, last = _book(torch, N, 32), _book(torch, N, 33)
    want, got = (torch.zeros(N, device="cuda:0") for _ in range(2))
    torch.cuda.synchronize()
    with Context(0, 1) as ctx:
        if shape:
            ctx.set_tune(*shape)
        ctx.price_soa(*last, want, n=N, device=True)
        for _ in range(3):
            ctx.price_soa(*first, got, n=N, num_runs=2, device=True, asynchronous=True, graph=False)
            ctx.price_soa(*last, got, n=N, num_runs=2, device=True, asynchronous=True, graph=False)
            ctx.synchronize()
            assert torch.equal(want.view(torch.int32), got.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES[:3], ids=str)
def test_inputs_produced_on_the_context_stream(shape):
    torch = pytest.importorskip("torch")
    s, k, r, v, t, o = _book(torch, N, 34)
    want, got = (torch.zeros(N, device="cuda:0") for _ in range(2))
    torch.cuda.synchronize()
    with Context(0, 1) as ctx:
        if shape:
            ctx.set_tune(*shape)
        twice = s * 2
        torch.cuda.synchronize()
        ctx.price_soa(twice, k, r, v, t, o, want, n=N, device=True)
        made = torch.zeros_like(s)
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
            torch.mul(s, 2, out=made)
        ctx.price_soa(made, k, r, v, t, o, got, n=N, num_runs=2, device=True, asynchronous=True, graph=False)
        ctx.synchronize()
    assert torch.equal(want.view(torch.int32), got.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 40_001, 1_000_003])
def test_host_passes_launched_one_by_one(n):
    """The gathered book of a host call is there when its first pass reads it."""
    torch = pytest.importorskip("torch")
    with Context(0, n) as ctx:
        for seed in range(35, 40):
            book = books.generate(n, seed=seed)
            want = ctx.price_book(book)
            keep = [torch.from_numpy(np.ascontiguousarray(a)).pin_memory() for a in book.arrays()]
            for arrays in (book.arrays(), [a.numpy() for a in keep]):
                got = np.zeros(n, np.float32)
                ctx.price_soa(*arrays, got, num_runs=3, graph=False)
                assert np.array_equal(want.view(np.uint32), got.view(np.uint32))


@pytest.mark.gpu
def test_plain_books_after_a_call_that_writes_the_pool():
    torch = pytest.importorskip("torch")
    s, k, r, v, t, o = _book(torch, N, 41)
    segs = [(i, min(99_990, N - i)) for i in range(0, N, 100_000)]
    outs = []
    for wait in (True, False):
        x, y = (torch.zeros(N, device="cuda:0") for _ in range(2))
        torch.cuda.synchronize()
        with Context(0, 1) as ctx:
            ctx.set_tune(1, 128, 0, 2, 1)
            ctx.price_soa(s, k, r, v, t, o, x, n=N, device=True, asynchronous=True)
            if wait:
                ctx.synchronize()
            ctx.price_batch([s, x, r, v, t, o], y, N, segs, plain=True, num_runs=2, asynchronous=True)
            ctx.synchronize()
        outs.append((x, y))
    for one, two in zip(*outs):
        assert torch.equal(one.view(torch.int32), two.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("call", ["graph", "direct", "batch", "batch direct", "plain books"])
def test_prices_over_an_input(shape, call):
    """Each pass takes the prices of the one before it as its spot prices."""
    torch = pytest.importorskip("torch")
    s, k, r, v, t, o = _book(torch, N, 42)
    segs = [(i, min(1_000_000, N - i)) for i in range(0, N, 1_000_000)]
    one, two = s.clone(), s.clone()
    torch.cuda.synchronize()
    with Context(0, 1) as ctx:
        for _ in range(3):
            ctx.price_soa(one, k, r, v, t, o, one, n=N, device=True)
        if shape:
            ctx.set_tune(*shape)
        if call in ("graph", "direct"):
            ctx.price_soa(two, k, r, v, t, o, two, n=N, num_runs=3, device=True, graph=call == "graph")
        else:
            ctx.price_batch([two, k, r, v, t, o], two, N, segs, num_runs=3, plain=call == "plain books",
                            graph=call != "batch direct")
    assert torch.equal(one.view(torch.int32), two.view(torch.int32))
