"""Contexts of several shapes in one process: none changes what another one may do."""
import numpy as np
import pytest

import tp3

pytestmark = pytest.mark.gpu


def test_split_coupling_after_a_smaller_context():
    """The split coupling's shared-memory limit is the process's: a small context made later leaves
    a large one's as it was, for its own calls and for its autotuning."""
    L, LMAX, N, K = 18, 19, 4, 26  # 79 KB a block
    big = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(2)
    big.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = rng.normal(size=(2, K, LMAX * LMAX)) + 1j * rng.normal(size=(2, K, LMAX * LMAX))
    big.set_mode(tp3.TP3_MODE_TC_BF16X3)
    big.set_coupling(1)
    want = big.energy_batch(c)
    small = tp3.calculate_basis(2, 3, 4, 2)
    assert np.array_equal(big.energy_batch(c), want)
    assert any(form == 1 for _, form, _, _ in big.autotune(2))
    small.close()
    big.close()
