"""The FP64 gradient elements' weights formed in integers (weights64 of
euler_fp64.cuh, compiled for the host) against exact ones: no further from
them than the FP64 operations that they replace (weights64_plain)."""

import ctypes
from decimal import Decimal, localcontext

import numpy as np
import pytest

from _device_host import library

CODE = r"""
using namespace scg::dev;
template <int N, int ND>
static int weights(double const * g, double acfl, double sigma0, double * wi, double * wp)
{
    double const ts = mu(mu(acfl, double(N - 1)), recip(sigma0));
    unsigned long long r[N];
    int h[N];
    double sq[N];
    bool fixed = cap_in_range(ts);
    for (int k = 0; k < N; ++k)
    {
        fixed = inverse_norm<ND>(g + k * ND, r[k], h[k]) && fixed;
        sq[k] = Tiny<double>::AZ;
        for (int d = 0; d < ND; ++d)
            sq[k] = fm(g[k * ND + d], g[k * ND + d], sq[k]);
    }
    int const fp = weights64_plain<N>(sq, acfl, sigma0, wp) ? 1 : 0;
    return fixed ? fp + (weights64<N>(r, h, ts, wi) ? 2 : 0) : 4;
}
extern "C" int weights(int n, double const * g, double acfl, double sigma0, double * wi, double * wp)
{
    return n == 3   ? weights<3, 2>(g, acfl, sigma0, wi, wp)
           : n == 4 ? weights<4, 3>(g, acfl, sigma0, wi, wp)
           : n == 6 ? weights<6, 3>(g, acfl, sigma0, wi, wp)
                    : weights<8, 3>(g, acfl, sigma0, wi, wp);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = library(tmp_path_factory.mktemp("weights"), CODE, ("euler_fp64.cuh",))
    p, d = ctypes.c_void_p, ctypes.c_double
    out.weights.argtypes = [ctypes.c_int, p, d, d, p, p]
    return out


def _exact(g, acfl, sigma0):
    """The reference's W-1/2 weights with the W-3/4 cap
    (euler_gradient.cpp:60-108) in 45 digits, and whether the cap fires."""
    tiny = Decimal(1e-200)
    n = Decimal(len(g))
    w = [1 / (sum(Decimal(float(x)) ** 2 for x in row) + tiny).sqrt()
         for row in g]
    total = sum(w)
    dev = [x / total - 1 / n for x in w]
    cap = min((1 - 1 / n) / (max(max(dev), 0) + tiny),
              (1 / n) / (tiny - min(min(dev), 0)))
    sigma = Decimal(sigma0) / Decimal(acfl)
    return [1 / n + min(cap, sigma) * d for d in dev], cap < sigma


# sigma0: the default, whose weights spread or are capped, to one at which they
# all but equal 1/N; spread: of the elements' gradients about a common one.
@pytest.mark.parametrize("n", [3, 4, 6, 8])
@pytest.mark.parametrize("sigma0", [3.0, 0.05, 1e-3])
@pytest.mark.parametrize("spread", [1e-8, 1.0, 1e3])
def test_weights_are_no_less_exact_than_in_fp64(lib, n, sigma0, spread):
    """In units of 2^-53.  A weight is one number rounded to the nearest from a
    fixed point of 2^-59 with an error of a few of its units: so its mean error
    is at most FP64's and a tenth (six units), and the sum of the weights, whose
    N roundings are unbiased, is one to a quarter of a unit on average."""
    rng = np.random.default_rng(n)
    ndim = 2 if n == 3 else 3
    err, sums = [], []
    wi, wp = np.empty(n), np.empty(n)
    with localcontext() as ctx:
        ctx.prec = 45
        for _ in range(300):
            g = rng.normal(size=(1, ndim)) + spread * rng.normal(size=(n, ndim))
            g = np.ascontiguousarray(g)
            acfl = float(rng.uniform(0.05, 1.0))
            got = lib.weights(n, g.ctypes.data, acfl, sigma0, wi.ctypes.data,
                              wp.ctypes.data)
            want, fires = _exact(g, acfl, sigma0)
            assert got == (3 if fires else 0)
            err.append([max(abs(Decimal(float(a)) - e)
                            for a, e in zip(w, want)) * 2 ** 53
                        for w in (wi, wp)])
            sums.append(float((sum(Decimal(float(a)) for a in wi) - 1)
                              * 2 ** 53))
    mine, fp64 = np.array(err, dtype="float64").mean(axis=0)
    assert mine <= fp64 + 0.1, (mine, fp64)
    assert abs(np.mean(sums)) <= 0.25, np.mean(sums)
