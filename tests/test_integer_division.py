"""The FP64 reciprocals, quotients, products and reciprocal roots formed in
integers (divide.cuh), compiled for the host and compared with exact ones, and
the same operands on the device.  The approximations that only the GPU has are
stood for by correctly rounded ones moved by up to two FP32 ulps (the hardware's
are within one)."""

import ctypes
from fractions import Fraction

import numpy as np
import pytest

from _device_host import library

CODE = r"""
using namespace scg::dev;
extern "C"
{
void quotients(double const * x, double const * d, double * q, int64_t n)
{
    for (int64_t i = 0; i < n; ++i)
        q[i] = div_fix(x[i], d[i], rcp_fix(d[i]));
}
void products(double const * a, double const * b, double * p, int64_t n)
{
    for (int64_t i = 0; i < n; ++i)
        p[i] = mul_int(a[i], b[i]);
}
void reciprocals(double const * d, double * r, int64_t n)
{
    for (int64_t i = 0; i < n; ++i)
        r[i] = recip(d[i]);
}
void roots(double const * x, double * r, int64_t n)
{
    for (int64_t i = 0; i < n; ++i)
        r[i] = rsq(x[i]);
}
uint64_t rcp_word(double d)
{
    return rcp_sig(static_cast<unsigned>(__double2hiint(d)), static_cast<unsigned>(__double2loint(d)));
}
uint64_t seed_word(double d)
{
    return seed24(seed_rcp(sig_top(static_cast<unsigned>(__double2hiint(d)), static_cast<unsigned>(__double2loint(d)))));
}
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = library(tmp_path_factory.mktemp("division"), CODE)
    for name in ("rcp_word", "seed_word"):
        getattr(lib, name).argtypes = [ctypes.c_double]
        getattr(lib, name).restype = ctypes.c_uint64
    return lib


def _double(sig, e, sign=0):
    return (sig | e.astype("uint64") << np.uint64(52)
            | np.uint64(sign) << np.uint64(63)).view("float64")


def _pairs():
    """x and d of every exponent, their quotients' exponents clustered where
    the code branches (a quotient of significands below one, the least and the
    largest normal numbers), significands at random, all ones, one bit, equal,
    and numerators next to a quotient half-way between two doubles; zeros,
    subnormals, infinities and NaN."""
    rng = np.random.default_rng(17)
    n = 1 << 17
    sig = rng.integers(0, 1 << 52, (5, 2, n), dtype=np.uint64)
    top = np.uint64((1 << 52) - 1)
    sig[1, 1] = top - (sig[1, 1] & np.uint64(3))
    sig[2, 1] = np.uint64(1) << (sig[2, 1] % np.uint64(52))
    sig[3, 1] = sig[3, 0] - np.minimum(sig[3, 0], rng.integers(0, 3, n, dtype=np.uint64))
    ed = rng.integers(1, 2047, (5, n))
    near = rng.choice([1, 1023, 2045], (5, n)) + rng.integers(-2, 4, (5, n))
    ex = np.where(rng.random((5, n)) < 0.7, ed - 1023 + near,
                  rng.integers(1, 2047, (5, n)))
    ok = (ex >= 1) & (ex <= 2046)
    ed = np.where(ok, ed, 1023)
    ex = np.clip(np.where(ok, ex, near), 1, 2046)
    # m d for m half-way between two doubles, rounded: a quotient next to m.
    m = 1.0 + (2 * (sig[4, 0] >> np.uint64(1)) + np.uint64(1)).astype("float64") * 2.0 ** -53
    sig[4, 0] = (m * (1.0 + sig[4, 1] * 2.0 ** -52)).view("uint64") & top
    sign = rng.integers(0, 2, (2, 5 * n), dtype=np.uint64) << np.uint64(63)
    x = _double(sig[:, 0], ex).ravel().view("uint64") | sign[0]
    d = _double(sig[:, 1], ed).ravel().view("uint64") | sign[1]
    special = np.array([0.0, -0.0, 1.0, -1.5, 5e-324, -1e-310, 2.0 ** -1022,
                        np.finfo(float).max, np.inf, -np.inf, np.nan])
    sx, sd = np.meshgrid(special, special)
    return (np.concatenate([x.view("float64"), sx.ravel()]),
            np.concatenate([d.view("float64"), sd.ravel()]))


def _same(got, want):
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.int64),
                                  want[~nan].view(np.int64))


def _run(f, *arrays):
    f(*[ctypes.c_void_p(a.ctypes.data) for a in arrays],
      ctypes.c_int64(arrays[0].size))


@pytest.mark.parametrize("shift", [-2, -1, 0, 1, 2])
def test_quotients_and_products_are_the_ieee_ones(host, shift):
    host.set_seed_shift(shift)
    x, d = _pairs()
    out = np.empty_like(x)
    with np.errstate(all="ignore"):
        _run(host.quotients, x, d, out)
        _same(out, x / d)
        _run(host.products, x, d, out)
        _same(out, x * d)


@pytest.mark.parametrize("shift", [-2, -1, 0, 1, 2])
def test_reciprocal_words(host, shift):
    """rcp_sig: the seed's residual is below 2^-21, as its 32-bit square needs,
    and the word within 2^-58 of 2^62 / m; recip and rsq round what they have
    within 0.52 ulp."""
    host.set_seed_shift(shift)
    rng = np.random.default_rng(3)
    sig = rng.integers(0, 1 << 52, 3000, dtype=np.uint64)
    sig[:600] = np.uint64((1 << 52) - 1) - np.arange(600, dtype=np.uint64)
    sig[600:1200] = np.arange(600, dtype=np.uint64)
    d = _double(sig, np.full(3000, 1023))
    for v, s in zip(d.tolist(), sig.tolist()):
        m = s | 1 << 52
        assert abs((1 << 76) - m * host.seed_word(v)) < 1 << 55
        assert abs(host.rcp_word(v) - Fraction(1 << 114, m)) <= 16
    r, q = np.empty_like(d), np.empty_like(d)
    d *= np.exp2(rng.integers(-1000, 1000, 3000).astype("float64"))
    _run(host.reciprocals, d, r)
    _run(host.roots, d, q)
    for v, rv, qv in zip(d.tolist(), r.tolist(), q.tolist()):
        ulp = Fraction(np.spacing(rv))
        assert abs(Fraction(rv) * Fraction(v) - 1) <= Fraction(52, 100) * ulp * Fraction(v)
        # |q - x^-1/2| <= h: (q - h)^2 <= 1 / x <= (q + h)^2.
        h = Fraction(52, 100) * Fraction(np.spacing(qv))
        assert (Fraction(qv) - h) ** 2 <= 1 / Fraction(v) <= (Fraction(qv) + h) ** 2


@pytest.mark.gpu
def test_quotients_and_products_on_the_device():
    from solvcon_gb300._lib import check, lib, ptr
    x, d = _pairs()
    q, qdiv, r, p = (np.empty_like(x) for _ in range(4))
    check(lib.scg_divide_check(ptr(x), ptr(d), ptr(q), ptr(qdiv), ptr(r), x.size))
    check(lib.scg_product_check(ptr(x), ptr(d), ptr(p), x.size))
    with np.errstate(all="ignore"):
        _same(q, x / d)
        _same(qdiv, x / d)
        _same(p, x * d)
        want = 1.0 / d
    inside = (np.abs(d) >= 2.0 ** -1022) & (np.abs(d) < 2.0 ** 1022)
    gap = np.abs(r[inside].view(np.int64) - want[inside].view(np.int64))
    assert gap.max() <= 1
    _same(r[~inside], want[~inside])
