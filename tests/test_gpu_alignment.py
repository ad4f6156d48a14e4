"""Arrays that are not aligned to their elements are a status, before anything is
launched."""
import numpy as np
import pytest

from p3arsec_gb300 import BsgError, Context, books
from p3arsec_gb300.abi import Server

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MISALIGNED = -6


def test_doubles_off_their_alignment_are_refused():
    """An array of doubles four bytes off is a status before anything is launched
    (the kernel copies and stores eight bytes at a time); four bytes are enough
    for the types."""
    n = 100
    book = books.generate(n + 2, seed=16)
    cols = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in book.arrays()]
    wide = [c.double() for c in cols[:5]] + [cols[5]]
    out = torch.full((n + 2,), -1.0, device="cuda:0", dtype=torch.float64)
    torch.cuda.synchronize()
    with Context(0, 1) as ctx:
        at = [x.data_ptr() for x in wide + [out]]
        for i in (0, 1, 2, 3, 4, 6):
            ptrs = list(at)
            ptrs[i] += 4
            for asynchronous in (False, True):
                with pytest.raises(BsgError) as e:
                    ctx.price_soa_f64(*ptrs, n=n, device=True, asynchronous=asynchronous)
                assert e.value.status == MISALIGNED
        with pytest.raises(BsgError) as e:
            ctx.price_fp64(*[x.data_ptr() for x in cols], out.data_ptr() + 4, n=n, device=True)
        assert e.value.status == MISALIGNED
        assert ctx.launches == 0
        ctx.price_soa_f64(*at[:5], at[5] + 4, at[6], n=n, device=True)
        ctx.price_soa_f64(*[p + 8 for p in at[:5]], at[5] + 4, at[6] + 8, n=n, device=True)
        assert ctx.launches == 2


@pytest.mark.parametrize("kind", [dict(fused=False), dict(fused=True), dict(persistent=True)], ids=str)
def test_requests_off_their_alignment_are_refused(kind):
    """The serving kernels read the caller's arrays in place; the plain loop copies
    them, from wherever they begin."""
    n = 100
    book = books.generate(n, seed=17)
    keep = [torch.zeros(n + 1).pin_memory() for _ in range(7)]
    bytes_of = [k.numpy().view(np.uint8) for k in keep]
    at = [k.data_ptr() for k in keep]
    for b, a in zip(bytes_of, book.arrays()):
        b[:4 * n] = a.view(np.uint8)
    with Server(budget_bytes=1 << 24, **kind) as srv:
        for k in keep:
            srv.register(k.numpy())
        for i in range(7):
            with pytest.raises(BsgError) as e:
                srv.submit(*[p + 2 * (j == i) for j, p in enumerate(at)], n=n)
            assert e.value.status == MISALIGNED
        assert srv.wait(srv.submit(*at, n=n), timeout_s=60.0)[0] == 0
        want = keep[6].numpy()[:n].copy()
        assert srv.stats()["completed"] == 1
    for b in bytes_of[:6]:
        b[2:4 * n + 2] = b[:4 * n].copy()
    with Server(budget_bytes=1 << 24, plain=True) as srv:
        assert srv.wait(srv.submit(*[p + 2 for p in at], n=n), timeout_s=60.0)[0] == 0
    assert np.array_equal(bytes_of[6][2:4 * n + 2].view(np.uint32), want.view(np.uint32))
