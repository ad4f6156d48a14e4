"""Short synchronous device calls wait for a word that their kernel stores; the
asynchronous call of the same book goes the other way.  Same bits, nothing
written beside, and a synchronous call leaves nothing of an asynchronous one
before it unfinished."""
import numpy as np
import pytest

from p3arsec_gb300 import Context, books

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N_MAX = 1 << 18  # kFlagOptions


@pytest.mark.parametrize("n", [1, 3, 4, 511, 513, N_MAX // 2, N_MAX // 2 + 1, N_MAX, N_MAX + 1])
def test_short_device_calls(n):
    book = books.generate(n + 4, seed=14)
    cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in book.arrays()]
    wide = [c.double() for c in cols[:5]] + [cols[5]]
    with Context(0, 1) as ctx:
        for mode in ("fast", "sfu_ref", "libm_ref"):
            one, two = (torch.full((n + 4,), -1.0, device="cuda:0") for _ in range(2))
            torch.cuda.synchronize()
            ctx.price_soa(*cols, one, n=n, mode=mode, device=True, asynchronous=True)
            ctx.price_soa(*cols, two, n=n, mode=mode, device=True)
            assert torch.equal(one.view(torch.int32), two.view(torch.int32)), mode
            assert (two[n:] == -1).all()
            for lo in (1, 3):  # a slice: up to three options in front of the vectors
                two.fill_(-1)
                torch.cuda.synchronize()
                ctx.price_soa(*[c[lo:lo + n] for c in cols], two[lo:lo + n], n=n, mode=mode, device=True)
                ctx.price_soa(*[c[lo:lo + n] for c in cols], one[lo:lo + n], n=n, mode=mode, device=True,
                              asynchronous=True)
                ctx.synchronize()
                assert torch.equal(one[lo:lo + n].view(torch.int32), two[lo:lo + n].view(torch.int32)), (mode, lo)
                assert (two[:lo] == -1).all() and (two[lo + n:] == -1).all()
        one, two, three = (torch.full((n + 4,), -1.0, device="cuda:0", dtype=torch.float64) for _ in range(3))
        torch.cuda.synchronize()
        ctx.price_soa_f64(*wide, one, n=n, device=True, asynchronous=True)
        ctx.price_soa_f64(*wide, two, n=n, num_runs=2, device=True)
        ctx.price_fp64(*cols, three, n=n, device=True)
        assert torch.equal(one.view(torch.int64), two.view(torch.int64))
        assert torch.equal(one.view(torch.int64), three.view(torch.int64))
        assert (two[n:] == -1).all()


@pytest.mark.parametrize("count", [1, 3, 3000])
def test_batch_of_one_pass_waits_for_its_kernel(count):
    """The last block of a synchronous batch stores the word; calls in a row take
    their work counter from the table each uploads."""
    rng = np.random.default_rng(count)
    lens = rng.integers(0, 5000, count)
    lens[0] = 7
    gaps = rng.integers(0, 9, count)
    at = np.concatenate([[0], np.cumsum(lens + gaps)[:-1]])
    segs = [(int(o), int(l)) for o, l in zip(at, lens)]
    n = int(at[-1] + lens[-1]) + 1
    cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in books.generate(n, seed=15).arrays()]
    one, two = (torch.full((n,), -1.0, device="cuda:0") for _ in range(2))
    with Context(0, 1) as ctx:
        torch.cuda.synchronize()
        ctx.price_batch(cols, one, n, segs, num_runs=2)
        for _ in range(3):
            two.fill_(-1)
            torch.cuda.synchronize()
            ctx.price_batch(cols, two, n, segs)
            assert torch.equal(one.view(torch.int32), two.view(torch.int32))
