"""The scoring kernels' own logarithm and float conversions against extended precision and numpy."""
import numpy as np
import pytest

import tp3
from tp3 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def run():
    b = tp3.calculate_basis(2, 3, 4, 2)

    def call(op, x, dtype):
        x = np.ascontiguousarray(x)
        out = np.empty(x.size, dtype=dtype)
        _lib.check(tp3.load().tp3_selftest_scalar(b.ctx, op, x.size, x.ctypes.data, out.ctypes.data), b.ctx)
        return out

    yield call
    b.close()


def test_log_over_the_exponent_range(run):
    """Within 2^-53 |log x| + 2^-60 of the logarithm in extended precision: the rounding of the result,
    and of the reduced argument |r| < 2^-8 and its sum."""
    rng = np.random.default_rng(1)
    m = np.concatenate([rng.uniform(1.0, 2.0, 200), 1.0 + np.arange(129) / 128.0,  # interval ends and their
                        np.nextafter(1.0 + np.arange(1, 129) / 128.0, 0.0)])       # neighbours below
    m = m[(m >= 1.0) & (m < 2.0)]
    x = np.ldexp(m[None], np.arange(-1022, 1024)[:, None]).ravel()
    near = 1.0 + np.ldexp(1.0, -np.arange(1, 53))
    x = np.concatenate([x, near, 2.0 - near, [1.0, np.finfo(float).tiny, np.finfo(float).max, 0.75, 1.5,
                                              np.nextafter(0.75, 0), np.nextafter(1.5, 0)]])
    ref = np.log(x.astype(np.longdouble))
    err = np.abs(run(0, x, np.float64).astype(np.longdouble) - ref)
    assert (err <= np.ldexp(np.abs(ref), -53) + np.longdouble(2.0) ** -60).all()


def test_log_of_special_values(run):
    sub = np.array([5e-324, 1e-310, np.nextafter(np.finfo(float).tiny, 0.0)])
    np.testing.assert_allclose(run(0, sub, np.float64), np.log(sub), rtol=2.0**-51)  # an ulp either side
    got = run(0, np.array([0.0, np.inf, -1.0, np.nan]), np.float64)
    assert got[0] == -np.inf and got[1] == np.inf and np.isnan(got[2]) and np.isnan(got[3])


def _same_bits(a, b):
    t = np.uint32 if a.dtype == np.float32 else np.uint64
    nan = np.isnan(b)
    assert np.array_equal(np.isnan(a), nan) and np.array_equal(a.view(t)[~nan], b.view(t)[~nan])


def test_float_to_double_is_exact(run):
    e = np.arange(256, dtype=np.uint32) << 23
    frac = np.array([0, 1, 2, 0x2AAAAA, 0x400000, 0x7FFFFE, 0x7FFFFF], dtype=np.uint32)
    u = (e[:, None] | frac[None]).ravel()
    x = np.concatenate([u, u | np.uint32(0x80000000)]).view(np.float32)
    _same_bits(run(1, x, np.float64), x.astype(np.float64))


def test_double_to_float_rounds_to_nearest_even(run):
    """Ties in both directions, one unit beside a tie, carries into the next binade, overflow to
    infinity, subnormal results, zeros, infinities and NaN: numpy's conversion bit for bit."""
    rng = np.random.default_rng(2)
    e = np.arange(1, 2047, 3, dtype=np.uint64) << np.uint64(52)
    e = np.concatenate([e, np.arange(860, 1160, dtype=np.uint64) << np.uint64(52)])
    top = np.array([0, 1, 2, 3, 0x2AAAAA, 0x7FFFFE, 0x7FFFFF], dtype=np.uint64) << np.uint64(29)
    low = np.array([0, 1, 0x0FFFFFFF, 0x10000000, 0x10000001, 0x1FFFFFFF], dtype=np.uint64)
    u = (e[:, None, None] | top[None, :, None] | low[None, None, :]).ravel()
    r = rng.integers(0, 1 << 63, 20000, dtype=np.uint64)
    special = np.array([0.0, np.inf, np.nan, 3.4028235677973366e38, 3.4028235677973362e38, 1e39, 1e-46, 7e-46,
                        1.1754943508222875e-38, 1.1754942807573643e-38, 5e-324])
    x = np.concatenate([u, r]).view(np.float64)
    x = np.concatenate([x, special])
    x = np.concatenate([x, -x])
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        _same_bits(run(2, x, np.float32), x.astype(np.float32))
