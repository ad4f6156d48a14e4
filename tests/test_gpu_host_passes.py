"""Several passes over a short host book are one kernel that brings the book in,
makes the passes and writes the last one's prices to the host: the bits of a
device call, nothing written beside them, at its edges (two and four options a
thread, options left over at the end, arrays off the vector boundary)."""
import numpy as np
import pytest

from p3arsec_gb300 import Context, books

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
@pytest.mark.parametrize("n", [2, 8193, 155_648, 155_651, 311_296])
def test_host_passes(n, pinned):
    pad = 9
    book = books.generate(n + pad, seed=8)
    with Context(0, n + pad) as ctx:
        for mode, lo in (("fast", 0), ("sfu_ref", 1), ("libm_ref", 2)):
            dev = [torch.from_numpy(a[lo:lo + n].copy()).cuda() for a in book.arrays()]
            out = torch.zeros(n, device="cuda:0")
            torch.cuda.synchronize()
            ctx.price_soa(*dev, out, n=n, mode=mode, device=True)
            want = out.cpu().numpy()
            whole = np.empty(n + pad, np.float32)
            arrays = [np.ascontiguousarray(a) for a in book.arrays()]
            if pinned:
                keep = [torch.from_numpy(a).pin_memory() for a in arrays + [whole]]
                arrays, whole = [k.numpy() for k in keep[:6]], keep[6].numpy()
            for runs in (2, 5, 100):
                whole[:] = -1
                ctx.price_soa(*[a[lo:lo + n] for a in arrays], whole[lo:lo + n], num_runs=runs, mode=mode)
                assert np.array_equal(whole[lo:lo + n].view(np.uint32), want.view(np.uint32)), (mode, runs)
                assert (whole[:lo] == -1).all() and (whole[lo + n:] == -1).all()


@pytest.mark.parametrize("n", [(1 << 17) - 1, 1 << 17, (1 << 17) + 1025, 400_007])
def test_pageable_book_in_two_launches(n):
    """From 2^17 options a pageable book's first eighth is priced while the rest
    of its pages are made present: the bits of a device call at the seam and at
    the ends, for arrays off the vector boundary too, nothing written beside."""
    pad = 9
    book = books.generate(n + pad, seed=9)
    arrays = [np.ascontiguousarray(a) for a in book.arrays()]
    with Context(0, n + pad) as ctx:
        for mode, lo in (("fast", 0), ("libm_ref", 3), ("fast", 1)):
            dev = [torch.from_numpy(a[lo:lo + n].copy()).cuda() for a in arrays]
            out = torch.zeros(n, device="cuda:0")
            torch.cuda.synchronize()
            ctx.price_soa(*dev, out, n=n, mode=mode, device=True)
            whole = np.full(n + pad, -1, np.float32)
            ctx.price_soa(*[a[lo:lo + n] for a in arrays], whole[lo:lo + n], mode=mode)
            assert np.array_equal(whole[lo:lo + n].view(np.uint32), out.cpu().numpy().view(np.uint32)), mode
            assert (whole[:lo] == -1).all() and (whole[lo + n:] == -1).all()


@pytest.mark.parametrize("n", [1, 63, 77_824, 77_825, 155_648, 155_649])
def test_passes_of_one_option_in_pairs(n):
    """Up to 512 options an SM (152) a thread owns one option and evaluates its
    passes two at a time: whatever their number, from any alignment, the bits of
    one pass."""
    book = books.generate(n + 3, seed=10)
    with Context(0, 1) as ctx:
        for mode, lo in (("fast", 0), ("sfu_ref", 3), ("libm_ref", 1)):
            dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda()[lo:lo + n] for a in book.arrays()]
            want, got = (torch.full((n + 3,), -1.0, device="cuda:0") for _ in range(2))
            torch.cuda.synchronize()
            ctx.price_soa(*dev, want[lo:lo + n], n=n, mode=mode, device=True)
            for runs in (2, 3, 4, 5, 9):
                got.fill_(-1)
                torch.cuda.synchronize()
                ctx.price_soa(*dev, got[lo:lo + n], n=n, num_runs=runs, mode=mode, device=True)
                assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (mode, lo, runs)
