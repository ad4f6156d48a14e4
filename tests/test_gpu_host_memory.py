"""Host calls through every route the context has for them -- its pinned
staging, the caller's pinned arrays in place, and copies -- at the sizes where
one takes over from another, with slices that are not vector-aligned.  Every
route evaluates the same operations: the prices are compared bit for bit with
device-pointer calls."""
import numpy as np
import pytest

from p3arsec_gb300 import Context, books

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STAGE, GATHER = 8192, 1 << 21  # kStageOptions, kGatherOptions
N_MAX = GATHER + 9


@pytest.fixture(scope="module")
def ctx():
    from p3arsec_gb300 import build as b
    b.build()
    c = Context(0, N_MAX)
    yield c
    c.close()


@pytest.fixture(scope="module")
def book():
    return books.generate(N_MAX + 8, seed=5)


def _want(ctx, book, lo, n, mode):
    arrays = [torch.from_numpy(a[lo:lo + n].copy()).cuda() for a in book.arrays()]
    out = torch.zeros(n, device="cuda:0")
    torch.cuda.synchronize()
    ctx.price_soa(*arrays, out, n=n, mode=mode, device=True)
    return out.cpu().numpy()


@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
@pytest.mark.parametrize("n", [1, 7, 64, 1001, STAGE, STAGE + 1, 100_003, GATHER, GATHER + 1])
def test_every_route(ctx, book, n, pinned):
    for mode, lo in (("fast", 0), ("libm_ref", 3), ("fast", 5)):
        if pinned:
            keep = [torch.from_numpy(a).pin_memory() for a in book.arrays()]
            keep.append(torch.full((N_MAX + 8,), -1.0).pin_memory())
            arrays = [k.numpy()[lo:lo + n] for k in keep]
            whole = keep[6].numpy()
        else:
            whole = np.full(N_MAX + 8, -1.0, np.float32)
            arrays = [a[lo:lo + n] for a in book.arrays()] + [whole[lo:lo + n]]
        want = _want(ctx, book, lo, n, mode)
        for runs in (1, 3):
            whole[:] = -1
            ctx.price_soa(*arrays, num_runs=runs, mode=mode)
            assert np.array_equal(whole[lo:lo + n].view(np.uint32), want.view(np.uint32)), (mode, runs)
            assert (whole[:lo] == -1).all() and (whole[lo + n:] == -1).all()


@pytest.mark.parametrize("n", [5000, 200_000])
def test_pinned_prices_over_an_input(ctx, book, n):
    """Prices that overwrite the spot prices, shifted by one option: the call
    reads every input before it writes, as its copies did."""
    keep = [torch.from_numpy(a[:n + 1]).pin_memory() for a in book.arrays()]
    arrays = [k.numpy()[:n] for k in keep]
    want = _want(ctx, book, 0, n, "fast")
    ctx.price_soa(*arrays, keep[0].numpy()[1:], n=n)
    assert np.array_equal(keep[0].numpy()[1:].view(np.uint32), want.view(np.uint32))


def test_read_only_file_mappings(ctx, book, tmp_path):
    """Inputs mapped read-only from files, prices in a fresh allocation whose
    pages nobody has touched."""
    n = 150_001
    arrays = []
    for i, a in enumerate(book.arrays()):
        a[:n].tofile(tmp_path / f"{i}.bin")
        arrays.append(np.memmap(tmp_path / f"{i}.bin", dtype=a.dtype, mode="r"))
    want = _want(ctx, book, 0, n, "fast")
    for runs in (1, 2):
        out = np.empty(n, np.float32)
        ctx.price_soa(*arrays, out, num_runs=runs)
        assert np.array_equal(out.view(np.uint32), want.view(np.uint32))


def test_wrong_host_arrays_are_refused(ctx, book):
    s, k, r, v, t, o = (a[:100] for a in book.arrays())
    out = np.zeros(100, np.float32)
    for bad in ((s.astype(np.float64), k, r, v, t, o, out), (s, k[:99], r, v, t, o, out),
                (s, k, r, v, t, o.astype(np.int64), out), (np.repeat(s, 2)[::2], k, r, v, t, o, out),
                (s, k, r, v, list(t), o, out), (s, k, r, v, t, o.view(np.float32), out)):
        with pytest.raises(TypeError):
            ctx.price_soa(*bad, n=100)


def test_host_and_asynchronous_calls_in_turn(ctx, book):
    """Staged calls between pipelined ones and asynchronous device calls."""
    n = 20_000
    arrays = [a[:n] for a in book.arrays()]
    want = _want(ctx, book, 0, n, "fast")
    dev = [torch.from_numpy(a.copy()).cuda() for a in arrays]
    dout = torch.zeros(n, device="cuda:0")
    torch.cuda.synchronize()
    piped = [np.zeros(n, np.float32) for _ in range(3)]
    for p in piped:
        small = np.zeros(50, np.float32)
        ctx.price_soa(*dev, dout, n=n, device=True, asynchronous=True)
        ctx.price_soa(*arrays, p, asynchronous=True)
        ctx.price_soa(*[a[:50] for a in arrays], small)
        assert np.array_equal(small.view(np.uint32), want[:50].view(np.uint32))
    ctx.synchronize()
    for p in piped + [dout.cpu().numpy()]:
        assert np.array_equal(p.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("n", [1, 16, STAGE, STAGE + 1, 200_000])
def test_device_memory_without_the_device_flag(ctx, book, n):
    """A C caller that leaves BSG_DEVICE_PTRS out has its arrays copied by the
    driver, wherever they are: every array in device memory, and each one alone."""
    arrays = [np.ascontiguousarray(a[:n]) for a in book.arrays()] + [np.zeros(n, np.float32)]
    want = _want(ctx, book, 0, n, "fast")
    dev = [torch.from_numpy(a).cuda() for a in arrays]
    torch.cuda.synchronize()
    for which in [set(range(7))] + [{i} for i in range(7)]:
        ptrs = [dev[i].data_ptr() if i in which else arrays[i].ctypes.data for i in range(7)]
        for runs in (1, 3):
            arrays[6][:] = -1
            dev[6].fill_(-1)
            torch.cuda.synchronize()
            assert ctx.lib.bsg_price_soa(ctx.h, *ptrs, n, runs, 0) == 0
            got = dev[6].cpu().numpy() if 6 in which else arrays[6]
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (which, runs)
    dev[6].fill_(-1)
    torch.cuda.synchronize()
    assert ctx.lib.bsg_BlkSchlsEqEuroNoDiv(dev[6].data_ptr(), n, *[d.data_ptr() for d in dev[:6]], 0.0) == 0
    assert np.array_equal(dev[6].cpu().numpy().view(np.uint32), want.view(np.uint32))
