"""One context, several modes and coupling forms in turn: each leaves the operands of the angular
stage in a layout of its own, and what an earlier call left beside the columns of the present one,
non-finite values included, must not reach its results."""
import numpy as np
import pytest

import tp3

pytestmark = pytest.mark.gpu

BF16, TF32, PLAIN = tp3.TP3_MODE_TC_BF16X3, tp3.TP3_MODE_TC_TF32X3, tp3.TP3_MODE_PLAIN_FP32


def _world(lam):
    L, LMAX, N, K, n = 6, 7, 6, 9, 3
    b = tp3.calculate_basis(L, LMAX, N, K, lam, 0.05 if lam else 0.0)
    assert b.n_lt % 16  # there are padding columns
    rng = np.random.default_rng(8)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = rng.normal(size=(n, K, LMAX * LMAX)) + 1j * rng.normal(size=(n, K, LMAX * LMAX))
    c[:, :, 0] += 8.0
    b.set_mode(TF32)  # operands of the wider type from the start: no reallocation in between
    b.reserve(n)
    return b, c


def _results(b, c):
    out = b.energy_batch(c), b.c3_raw(c[1]), b.energy_batch(c[:1])
    assert all(np.isfinite(x).all() for x in out)
    return out


@pytest.mark.parametrize("bad", [1e30, np.inf, np.nan])
def test_plain_after_a_nonfinite_tf32_batch(bad):
    """TF32 mode leaves T order-major in the buffer that the plain path reads by rows."""
    b, c = _world(0.0)
    b.set_mode(PLAIN)
    want = _results(b, c)
    b.set_mode(TF32)
    b.energy_batch(c * bad)
    b.set_mode(PLAIN)
    for got, ref in zip(_results(b, c), want):
        assert np.array_equal(got, ref)
    b.close()


FORMS = [(BF16, 9), (BF16, 0), (BF16, 7), (TF32, 9), (TF32, 0), (PLAIN, 0)]


@pytest.mark.parametrize("lam", [0.0, 1.7])
@pytest.mark.parametrize("bad", [1e30, np.inf, np.nan])
def test_every_form_after_a_nonfinite_batch_of_another(lam, bad):
    """A batch whose T overflows (or is NaN) in one (mode, form), then clean proposals in another."""
    b, c = _world(lam)

    def select(mode, form):
        b.set_mode(mode)
        b.set_coupling(form)

    want = {}
    for f in FORMS:
        select(*f)
        want[f] = _results(b, c)
    for dirty in FORMS:
        for f in FORMS:
            select(*dirty)
            b.energy_batch(c * bad)
            select(*f)
            for got, ref in zip(_results(b, c), want[f]):
                assert np.array_equal(got, ref), (dirty, f)
    b.close()
