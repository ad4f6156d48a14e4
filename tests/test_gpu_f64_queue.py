"""Double prices: the options that the fixed-point evaluation leaves to the
double one pass through a queue per block.  However many there are and wherever
they stand, an option gets the bits it gets in a book of its own kind."""
import numpy as np
import pytest

from p3arsec_gb300 import books

pytestmark = pytest.mark.gpu


def kinds():
    """97 options, every third outside the fixed-point domain (v^2 t < 2^-52)."""
    b = books.generate(97, seed=21, dist="tails")
    s, k, r, v, t = (np.asarray(getattr(b, n)).astype(np.float64)
                     for n in ("sptprice", "strike", "rate", "volatility", "otime"))
    v[::3] = 1e-9
    return [s, k, r, v, t, np.asarray(b.otype).astype(np.int32)]


# 32 options a warp, a block per SM (152), 1024 queue entries a block
@pytest.mark.parametrize("n", [1, 31, 33, 4863, 4865, 400_003])
@pytest.mark.parametrize("which", ["few", "third", "all"])
def test_bits_do_not_depend_on_the_queue(gpu_ctx, n, which):
    base = kinds()
    alone = np.zeros(97)
    gpu_ctx.price_soa_f64(*base, alone)
    if which == "all":
        idx = 3 * (np.arange(n) % 33)
    else:
        idx = np.arange(n) % 97
        if which == "few":
            idx = np.where((idx % 3 == 0) & (np.arange(n) % 40 != 0), idx + 1, idx) % 97
    out = np.zeros(n)
    gpu_ctx.price_soa_f64(*[np.ascontiguousarray(a[idx]) for a in base], out)
    assert np.array_equal(out.view(np.uint64), alone[idx].view(np.uint64))
    f32 = [np.ascontiguousarray(a[idx].astype(np.float32)) for a in base[:5]]
    got, ref = np.zeros(n), np.zeros(97)
    gpu_ctx.price_fp64(*f32, np.ascontiguousarray(base[5][idx]), got)
    gpu_ctx.price_fp64(*[a.astype(np.float32) for a in base[:5]], base[5], ref)
    assert np.array_equal(got.view(np.uint64), ref[idx].view(np.uint64))
