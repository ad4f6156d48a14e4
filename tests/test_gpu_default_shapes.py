"""The shapes a context that was never tuned takes for device books: slices
that start anywhere in a book, several passes of a short book in one launch,
and books whose prices overwrite an input.  Every shape evaluates the same
operations, so the prices are compared bit for bit with one pass of the
scalar kernel (arrays that are not equally aligned)."""
import numpy as np
import pytest

from p3arsec_gb300 import Context, books

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SMS = 152
MODES = ("fast", "sfu_ref", "libm_ref")


@pytest.fixture(scope="module")
def ctx():
    from p3arsec_gb300 import build as b
    b.build()
    c = Context(0, 1)
    yield c
    c.close()


def _device(book, offsets):
    out = []
    for a, o in zip(book.arrays(), offsets):
        t = torch.zeros(len(a) + o, dtype=torch.from_numpy(a).dtype, device="cuda:0")
        t[o:] = torch.from_numpy(a).cuda()
        out.append(t[o:])
    torch.cuda.synchronize()
    return out


def _price(ctx, arrays, n, offset, runs, mode):
    room = torch.full((n + 16,), -1.0, dtype=torch.float32, device="cuda:0")
    torch.cuda.synchronize()
    ctx.price_soa(*arrays, room[offset:offset + n], n=n, num_runs=runs, mode=mode, device=True)
    got = room.cpu().numpy()
    assert (got[:offset] == -1).all() and (got[offset + n:] == -1).all()
    return got[offset:offset + n].view(np.uint32)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n", [1, 2, 5, 7, 8, 9, 31, 64, 1023, SMS * 1024, SMS * 1024 + 3, SMS * 2048 - 1,
                               SMS * 2048 + 8, 700_001])
def test_every_offset_and_number_of_passes(ctx, n, mode):
    book = books.generate(n, seed=n)
    want = _price(ctx, _device(book, (0, 1, 2, 3, 1, 2)), n, 3, 1, mode)
    for offset in (0, 1, 3, 4, 7, 8):
        arrays = _device(book, (offset,) * 6)
        for runs in (1, 2, 5, 9):
            got = _price(ctx, arrays, n, offset, runs, mode)
            assert np.array_equal(got, want), (offset, runs)


@pytest.mark.parametrize("n", [1000, 400_000])
def test_prices_over_an_input(ctx, n):
    """Two passes whose prices overwrite the spot prices equal two calls of one."""
    book = books.generate(n, seed=3)
    a, b = _device(book, (0,) * 6), _device(book, (0,) * 6)
    ctx.price_soa(*a, a[0], n=n, num_runs=2, device=True)
    for _ in range(2):
        ctx.price_soa(*b, b[0], n=n, num_runs=1, device=True)
    assert torch.equal(a[0].view(torch.int32), b[0].view(torch.int32))


def test_large_books_of_each_shape(ctx):
    """Past half the L2, past 2.5 of it and past 6: ten passes against one."""
    for n in (3_000_001, 13_000_003, 30_000_000):
        arrays = books.generate_device(n, seed=n)
        torch.cuda.synchronize()
        one = torch.zeros(n, device="cuda:0")
        ten = torch.zeros(n, device="cuda:0")
        torch.cuda.synchronize()
        ctx.price_soa(*arrays, one, n=n, num_runs=1, device=True)
        ctx.price_soa(*arrays, ten, n=n, num_runs=10, device=True)
        assert torch.equal(one.view(torch.int32), ten.view(torch.int32))
