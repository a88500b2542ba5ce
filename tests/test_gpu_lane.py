"""The lane-owned coupling against the one-kernel pair coupling: both add every triple product
in the same order, so T, c3 and the energies are equal bit for bit, at shapes on either side
of the lane form's tiles: 32 shell pairs a unit, blocks of 8 and 16 shells k3, three orders a
task, 32 shells a coefficient row, quads of four m3, real-function and general coefficients."""
import numpy as np
import pytest

import tp3

pytestmark = pytest.mark.gpu

LANE, PAIR = 9, 0


def _coefficients(L, LMAX, K, n, real, seed):
    """n coefficient sets; c[l,-m] = (-1)^m conj c[l,m] when real."""
    from tp3.structure import seanindex0
    rng = np.random.default_rng(seed)
    c = np.zeros((n, K, LMAX * LMAX), dtype=np.complex128)
    for l in range(L + 1):
        for m in range(l + 1):
            v = (rng.normal(size=(n, K)) + 1j * rng.normal(size=(n, K)) * (m > 0)) / (1.0 + l)
            c[:, :, seanindex0(l, m, LMAX)] = v
            if m:
                c[:, :, seanindex0(l, -m, LMAX)] = (-1) ** m * np.conj(v)
    c[:, :, seanindex0(0, 0, LMAX)] += 4.0
    if not real:
        c += 0.1 * (rng.normal(size=c.shape) + 1j * rng.normal(size=c.shape))
    return c


@pytest.mark.parametrize("L,LMAX,N,K", [(0, 1, 2, 1), (2, 3, 4, 7), (4, 6, 6, 8), (6, 7, 8, 9), (10, 11, 8, 16),
                                        (8, 9, 8, 17), (12, 13, 10, 32), (6, 8, 6, 33), (4, 5, 4, 64), (18, 20, 8, 5),
                                        (30, 31, 4, 3)])
@pytest.mark.parametrize("real", [True, False])
def test_lane_form_equals_pair_form(L, LMAX, N, K, real):
    b = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(K)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = _coefficients(L, LMAX, K, 3, real, 10 * L + K)
    got = {}
    for form in (PAIR, LANE):
        b.set_mode(tp3.TP3_MODE_TC_BF16X3)
        b.set_coupling(form)
        T, c3, E = b.triple_products(c[0]), b.c3_raw(c[0]), b.energy_batch(c)
        b.set_mode(tp3.TP3_MODE_TC_TF32X3)
        got[form] = (T, c3, E, b.triple_products(c[1]), b.c3_raw(c[1]), b.energy_batch(c))
    for x, y in zip(got[PAIR], got[LANE]):
        assert np.isfinite(x).all() and np.array_equal(x, y)
    b.close()


def test_lane_form_mixed_and_ragged_batches():
    """One batch with real-function and general proposals; ragged limits with absent orders and
    shells: energies equal the pair form's."""
    import torch
    L, LMAX, N, K = 14, 15, 12, 21
    b = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(3)
    Ks = [K, 13, 16, 17]
    hists = [rng.uniform(0.5, 1.5, size=(N, 2 * N, k, k, k)) for k in Ks]
    b.set_histogram(hists[0])
    b.set_histograms(hists, Ks)
    c = _coefficients(L, LMAX, K, 6, True, 5)
    c[1::2] = _coefficients(L, LMAX, K, 3, False, 6)
    lkh = np.array([(14, 21, 0), (6, 13, 1), (12, 16, 2), (0, 1, 3), (8, 17, 3), (2, 9, 1)], dtype=np.int32)
    d_c = torch.from_numpy(c.view(np.float64).copy()).cuda()
    d_l = torch.from_numpy(lkh).cuda()
    got = {}
    for form in (PAIR, LANE):
        b.set_coupling(form)
        E, R = (torch.empty(6, dtype=torch.float64, device="cuda") for _ in range(2))
        b.energy_batch_device(6, d_c.data_ptr(), E.data_ptr())
        b.energy_batch_ragged_device(6, d_c.data_ptr(), d_l.data_ptr(), R.data_ptr())
        b.sync()
        got[form] = (E.cpu().numpy(), R.cpu().numpy())
    for x, y in zip(got[PAIR], got[LANE]):
        assert np.isfinite(x).all() and np.array_equal(x, y)
    b.close()


def test_lane_form_is_the_default():
    b = tp3.calculate_basis(8, 9, 8, 8)
    c = _coefficients(8, 9, 8, 1, True, 1)[0]
    T = b.triple_products(c)
    b.set_coupling(LANE)
    assert np.array_equal(T, b.triple_products(c))
    b.close()


@pytest.mark.parametrize("L,LMAX,N,K,n", [(0, 1, 2, 1, 1), (2, 3, 4, 5, 4), (6, 7, 6, 8, 5), (10, 12, 8, 9, 9),
                                          (12, 13, 10, 17, 13), (24, 25, 4, 6, 14)])
def test_fourier_pair_operand_equals_entry_sums(L, LMAX, N, K, n):
    """lambda != 0: H from mirrored entry pairs (lane form) against the sum over all entries
    (pair form), batches on either side of 4, 8 and 12 proposals a CTA."""
    b = tp3.calculate_basis(L, LMAX, N, K, 1.7, 0.05)
    rng = np.random.default_rng(L)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = _coefficients(L, LMAX, K, n, True, L + 1)
    if n > 1:
        c[1] = _coefficients(L, LMAX, K, 1, False, L + 2)[0]
    for mode in (tp3.TP3_MODE_TC_BF16X3, tp3.TP3_MODE_TC_TF32X3):
        got = {}
        b.set_mode(mode)
        for form in (PAIR, LANE):
            b.set_coupling(form)
            got[form] = (b.c3_raw(c[0]), b.energy_batch(c))
        for x, y in zip(got[PAIR], got[LANE]):
            assert np.isfinite(x).all() and np.array_equal(x, y)
    b.close()


@pytest.mark.parametrize("N", [2, 16, 18, 22, 24, 28, 32])
def test_grid_halves_and_batch_sizes(N):
    """Grids of Gu = N^2/2 points on either side of 128, 256 and 384, the widths of the persistent
    schedule's products; one proposal (tasks spread over small CTAs, a cluster sums the energy)
    against the same proposals in a batch of 160 (one CTA a sum) bit for bit, and against the
    per-tile schedule.  Both schedules add the same FP32 c3 and keep the sums compensated, so they
    differ by the rounding of the stored partials, 2^-24 each, of a slab's Qs log Sp and Sql with
    Qs = 1 and |log| below 70 (c3 is clamped at 1e-30): K^3 slabs of 2^-23 x 80."""
    L, LMAX, K, n = 6, 7, 9, 160
    b = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(N)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = _coefficients(L, LMAX, K, n, True, N)
    for mode in (tp3.TP3_MODE_TC_BF16X3, tp3.TP3_MODE_TC_TF32X3):
        b.set_mode(mode)
        b.set_coupling(LANE)
        E = b.energy_batch(c)
        assert np.isfinite(E).all()
        one = np.array([b.energy_batch(c[i:i + 1])[0] for i in (0, 75, n - 1)])
        assert np.array_equal(one, E[[0, 75, n - 1]])
        b.set_angular(tp3.TP3_ANGULAR_TILE)
        assert np.abs(b.energy_batch(c) - E).max() <= 2.0**-23 * 80 * K**3
        b.set_angular(tp3.TP3_ANGULAR_PERSISTENT)
    b.close()


@pytest.mark.parametrize("broken", [0.0, 1e-12, 1e-7])
def test_gather_takes_the_pair_forms_branch(broken):
    """Mirrored orders equal only to a part of the largest coefficient: below 1e-10 of it they
    count as a real function's, above as general ones, in both forms."""
    L, LMAX, N, K = 8, 9, 6, 11
    b = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(4)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = _coefficients(L, LMAX, K, 2, True, 9)
    from tp3.structure import seanindex0
    c[1, K - 1, seanindex0(4, -3, LMAX)] += broken * np.abs(c).max()
    got = {}
    b.set_mode(tp3.TP3_MODE_TC_BF16X3)
    for form in (PAIR, LANE):
        b.set_coupling(form)
        got[form] = (b.triple_products(c[1]), b.energy_batch(c))
    for x, y in zip(got[PAIR], got[LANE]):
        assert np.isfinite(x).all() and np.array_equal(x, y)
    b.close()


@pytest.mark.parametrize("L,N,K,n", [(12, 16, 16, 1), (12, 16, 16, 4), (18, 32, 26, 4)])
@pytest.mark.parametrize("mode", [tp3.TP3_MODE_TC_BF16X3, tp3.TP3_MODE_TC_TF32X3])
def test_general_coefficients_are_no_slower_than_in_the_pair_form(L, N, K, n, mode):
    """The default form takes general coefficients in runs of orders; a pass per order was slower than
    the one-kernel form, which has both signs of m3 in one pass."""
    import torch
    b = tp3.calculate_basis(L, L + 1, N, K)
    rng = np.random.default_rng(1)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    d_c = torch.from_numpy(_coefficients(L, L + 1, K, n, False, 4).view(np.float64).copy()).cuda()
    d_E = torch.empty(n, dtype=torch.float64, device="cuda")
    b.set_mode(mode)
    stream = torch.cuda.Stream()
    b.set_stream(stream.cuda_stream)
    best, E = {PAIR: 1e9, LANE: 1e9}, {}
    for rep in range(8):  # in turn
        for form in (PAIR, LANE):
            b.set_coupling(form)
            b.energy_batch_device(n, d_c.data_ptr(), d_E.data_ptr())
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record(stream)
            for _ in range(50):
                b.energy_batch_device(n, d_c.data_ptr(), d_E.data_ptr())
            e1.record(stream)
            b.sync()
            best[form] = min(best[form], e0.elapsed_time(e1))
            E[form] = d_E.cpu().numpy()
    assert np.array_equal(E[PAIR], E[LANE])
    assert best[LANE] <= best[PAIR], best
    b.set_stream(None)
    b.close()


@pytest.mark.parametrize("L,K", [(6, 12), (16, 17), (18, 26), (22, 9)])
@pytest.mark.parametrize("n", [1, 2, 40])
def test_runs_of_orders_equal_the_pair_form(L, K, n):
    """General coefficients, alone and beside real functions: balanced runs of one to three orders, some
    blocks in more runs than that (small L), passes spread over a block's CTAs (small n) or taken in
    turn by one (n = 40)."""
    LMAX, N = L + 1, 6
    b = tp3.calculate_basis(L, LMAX, N, K)
    rng = np.random.default_rng(n)
    b.set_histogram(rng.uniform(0.5, 1.5, size=(N, 2 * N, K, K, K)))
    c = _coefficients(L, LMAX, K, n, False, L)
    c[1::3] = _coefficients(L, LMAX, K, len(c[1::3]), True, K)
    got = {}
    for form in (PAIR, LANE):
        b.set_coupling(form)
        got[form] = (b.triple_products(c[0]), b.energy_batch(c))
    for x, y in zip(got[PAIR], got[LANE]):
        assert np.isfinite(x).all() and np.array_equal(x, y)
    b.close()


def test_form_in_use():
    """The lane-owned form is what a context starts with unless its shared memory does not fit (more
    than 64 shells); a forced form is the one reported."""
    b = tp3.calculate_basis(8, 10, 6, 8)
    assert b.coupling == LANE
    b.set_coupling(PAIR)
    assert b.coupling == PAIR
    for form in range(1, 10):
        try:
            b.set_coupling(form)
        except tp3.TP3Error:
            continue
        assert b.coupling == form
    b.close()
    b = tp3.calculate_basis(8, 9, 4, 70)
    assert b.coupling != LANE
    with pytest.raises(tp3.TP3Error):
        b.set_coupling(LANE)
    b.close()
