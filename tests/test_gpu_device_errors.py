"""A device wait that runs out is reported by the call it spoils, not by a later one."""
import numpy as np
import pytest

import tp3
from tp3 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["triple_products", "c3_raw", "energy_batch"])
def test_timeout_is_reported_by_the_synchronising_call(call):
    L, LMAX, N, K = 4, 5, 4, 3
    b = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(1)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = rng.normal(size=(K, LMAX * LMAX)) + 0j
    if call == "energy_batch":
        c = c[None]
    want = getattr(b, call)(c)
    assert tp3.load().tp3_selftest_timeout(b.ctx, 1_000_000) == 0
    with pytest.raises(tp3.TP3Error) as ei:
        getattr(b, call)(c)
    assert ei.value.status == _lib.TP3_ERR_TIMEOUT
    assert np.array_equal(getattr(b, call)(c), want)
    b.close()
