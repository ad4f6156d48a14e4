"""Host arrays that begin at any address, through the staging and the longer
routes: the prices of the same options in aligned arrays."""
import numpy as np
import pytest

from p3arsec_gb300 import books

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 100, 8192, 8193, 200_001])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_host_arrays_at_odd_addresses(gpu_ctx, n, off):
    book = books.generate(n, seed=off)
    odd = []
    for a in list(book.arrays()) + [np.zeros(n, np.float32)]:
        x = np.zeros(4 * n + 4, np.uint8)[off:off + 4 * n].view(a.dtype)
        x[:] = a
        odd.append(x)
    for runs in (1, 2):
        want = gpu_ctx.price_book(book, num_runs=runs)
        odd[6][:] = -1
        gpu_ctx.price_soa(*odd, num_runs=runs)
        assert odd[6].tobytes() == want.tobytes()
