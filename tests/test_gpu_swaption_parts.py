"""A swaption's paths are split into parts by the number of trials alone, and
the parts summed in an order of their own: its bits do not depend on what else
is priced, on whether the table travels with the launch or is copied first, or
on what the call before left behind."""
import numpy as np
import pytest

from p3arsec_gb300 import swaptions as S

pytestmark = pytest.mark.gpu


# one path, parts without paths, 256 parts (one group) and 264 (nine of 32), one
# and two paths a thread
@pytest.mark.parametrize("trials", [2, 33, 8192, 8193, 155_136, 155_137])
def test_bits_alone_and_among_others(gpu_ctx, oracle_lib, trials):
    few, many = S.generate(3, seed=11), S.generate(48, seed=12)
    mixed = many[:20] + few + many[20:]       # longest paths first inside
    p1, e1 = gpu_ctx.price_swaptions(few, trials)
    p2, e2 = gpu_ctx.price_swaptions(mixed, trials)
    for i in range(3):
        pa, ea = gpu_ctx.price_swaptions(few[i:i + 1], trials)
        assert pa[0] == p1[i] == p2[20 + i]
        assert np.array_equal([ea[0], e1[i]], [e1[i], e2[20 + i]], equal_nan=True)
    for _ in range(2):
        assert np.array_equal(gpu_ctx.price_swaptions(mixed, trials)[0], p2)
    want, _, _ = oracle_lib.swaptions_all(few, trials, 8)
    assert np.allclose(p1, want, rtol=1e-10, atol=1e-12)
