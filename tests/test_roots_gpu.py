"""The FP64 march's reciprocal roots and roots, formed on the integer pipe,
against correctly rounded ones."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operands():
    """Positive normal numbers over every exponent of both parities:
    significands at random, all ones, all zeros but one bit, perfect squares;
    and what the library functions take: zeros, subnormals, negative numbers,
    infinities and NaN."""
    rng = np.random.default_rng(5)
    n = 1 << 17
    e = rng.integers(1, 2047, n, dtype=np.uint64) << np.uint64(52)
    x = (rng.integers(0, 1 << 52, n, dtype=np.uint64) | e).view(np.float64)
    ones = (e[:4092] | np.uint64((1 << 52) - 1)).view(np.float64)
    every = np.arange(1, 2047, dtype=np.uint64) << np.uint64(52)
    low = (every | np.uint64(1)).view(np.float64)
    squares = rng.integers(1, 1 << 26, 4096).astype("float64") ** 2
    outside = np.array([0.0, -0.0, 5e-324, 1e-310, -1.0, -5e-324, np.inf,
                        -np.inf, np.nan])
    return np.concatenate([x, ones, every.view(np.float64), low, squares,
                           [1e-200, np.finfo(float).max, 2.0 ** -1022],
                           outside]), outside.size


def test_roots_within_one_ulp():
    """Both are within 0.52 ulp of the exact value, so each is the correctly
    rounded one or its neighbour; perfect squares are exact."""
    from solvcon_gb300._lib import check, lib, ptr
    x, nout = _operands()
    r, s = np.empty_like(x), np.empty_like(x)
    check(lib.scg_root_check(ptr(x), ptr(r), ptr(s), x.size))
    body = slice(0, x.size - nout)
    with np.errstate(all="ignore"):
        want_s = np.sqrt(x)
        want_r = (1 / np.sqrt(x.astype(np.longdouble))).astype("float64")
    for got, want in ((r, want_r), (s, want_s)):
        gap = np.abs(got[body].view(np.int64) - want[body].view(np.int64))
        assert gap.max() <= 1, x[body][gap > 1][:5]
    exact = want_s[body] ** 2 == x[body]
    exact &= want_s[body] == np.rint(want_s[body])
    assert (s[body][exact] == want_s[body][exact]).all()
    out = slice(x.size - nout, x.size)
    np.testing.assert_array_equal(s[out], want_s[out])
    np.testing.assert_allclose(r[out], want_r[out], rtol=3e-16)
