"""Served requests whose arrays start anywhere: slices 0 to 3 options past a
16-byte boundary (vector tiles from the boundary on), and arrays that are not
equally far from one, at the sizes around a tile and a vector.  Every path of
the loop gives the map's bits and writes nothing past a request."""
import numpy as np
import pytest

from p3arsec_gb300 import books
from p3arsec_gb300.abi import Server

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TILE = 2048


@pytest.mark.parametrize("kind", ["fused", "persistent", "unfused"])
def test_slices_at_every_offset(gpu_ctx, kind):
    sizes = [1, 2, 3, 4, 5, 7, 255, TILE - 1, TILE, TILE + 1, TILE + 3, 3 * TILE, 3 * TILE + 2, 20_011]
    pool_n = 4 * sum(n + 8 for n in sizes) + 64
    book = books.generate(pool_n, seed=21)
    keep = [torch.from_numpy(a).pin_memory() for a in book.arrays()]
    keep.append(torch.full((pool_n,), -1.0).pin_memory())
    pool = [k.numpy() for k in keep]
    want = gpu_ctx.price_book(book)
    with Server(0, budget_bytes=1 << 28, fused=kind != "unfused", persistent=kind == "persistent") as srv:
        for a in pool:
            srv.register(a)
        ids, spans, at = [], [], 0
        for off in range(4):
            for n in sizes:
                at = (at + 3) // 4 * 4 + off
                ids.append(srv.submit(*[a[at:at + n] for a in pool], n))
                spans.append((at, n))
                at += n + 2
        for i in ids:
            assert srv.wait(i, 20)[0] == 0
        out = pool[6]
        priced = np.zeros(pool_n, bool)
        for a, n in spans:
            assert np.array_equal(out[a:a + n].view(np.uint32), want[a:a + n].view(np.uint32)), (a, n)
            priced[a:a + n] = True
        assert (out[~priced] == -1).all()
        # arrays at different offsets from a boundary
        n = 5000
        arrays = [a[j:j + n] for j, a in enumerate(pool[:6])]
        got = pool[6][6:6 + n]
        assert srv.wait(srv.submit(*arrays, got, n), 20)[0] == 0
        mixed = gpu_ctx.price_book(books.Book(*[np.ascontiguousarray(a) for a in arrays]))
        assert np.array_equal(got.view(np.uint32), mixed.view(np.uint32))
