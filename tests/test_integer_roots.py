"""The FP64 root formed in integers (sqr_t of divide.cuh, compiled for the
host) is the IEEE root, whatever the GPU's approximation that it starts from
is within its stated error."""

import ctypes

import numpy as np
import pytest

from _device_host import library

CODE = r"""
extern "C" void roots(double const * x, double * s, int64_t n)
{
    for (int64_t i = 0; i < n; ++i)
        s[i] = scg::dev::sqr_t(x[i]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return library(tmp_path_factory.mktemp("roots"), CODE)


def operands():
    """Significands at random, of few bits, next to all ones and next to the
    squares of the halves between two 53-bit roots, over every exponent; and
    zeros, subnormals, negative numbers, infinities and NaN."""
    rng = np.random.default_rng(5)
    n = 1 << 18
    e = rng.integers(1, 2047, (4, n), dtype=np.uint64) << np.uint64(52)
    sig = rng.integers(0, 1 << 52, (4, n), dtype=np.uint64)
    sig[1] &= np.uint64(0xffffff8000000)
    sig[2] = np.uint64((1 << 52) - 1) - (sig[2] & np.uint64(1023))
    # (k + 1/2)^2 for a 53-bit k, cut to 53 bits, and its neighbours.
    k = rng.integers(1 << 52, 1 << 53, n).astype(object)
    m = [((2 * v + 1) ** 2 << 4) >> ((2 * v + 1) ** 2).bit_length() - 49
         for v in k]
    sig[3] = np.array([v & ((1 << 52) - 1) for v in m], dtype=np.uint64)
    sig[3] += rng.integers(0, 2, n, dtype=np.uint64)
    odd = np.array([((2 * v + 1) ** 2).bit_length() & 1 for v in k],
                   dtype=np.uint64)
    e[3] = (np.uint64(1024) - odd) << np.uint64(52)
    sig[3] &= np.uint64((1 << 52) - 1)
    out = np.array([0.0, -0.0, 5e-324, 1e-310, -1.0, -5e-324, np.inf, -np.inf,
                    np.nan, 2.0 ** -1022, np.finfo(float).max])
    return np.concatenate([(sig | e).view(np.float64).ravel(), out])


@pytest.mark.parametrize("shift", [-2, -1, 0, 1, 2])
def test_root_is_the_ieee_root(lib, shift):
    x = operands()
    s = np.empty_like(x)
    lib.set_seed_shift(shift)
    lib.roots(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(s.ctypes.data),
              ctypes.c_int64(x.size))
    with np.errstate(all="ignore"):
        want = np.sqrt(x)
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(s), nan)
    np.testing.assert_array_equal(s[~nan].view(np.int64),
                                  want[~nan].view(np.int64))


@pytest.mark.gpu
def test_root_on_the_device():
    from solvcon_gb300._lib import check, lib, ptr
    x = operands()
    r, s = np.empty_like(x), np.empty_like(x)
    check(lib.scg_root_check(ptr(x), ptr(r), ptr(s), x.size))
    with np.errstate(all="ignore"):
        want = np.sqrt(x)
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(s), nan)
    np.testing.assert_array_equal(s[~nan].view(np.int64),
                                  want[~nan].view(np.int64))
