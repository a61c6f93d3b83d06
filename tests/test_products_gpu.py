"""The 1D marches' FP64 products on the integer pipe: bit for bit the FP64
product, and large tubes and grids, which use them, bit for bit the small ones,
which do not."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs():
    """Random significands over every exponent (products in, at the edges of
    and beyond the normal range), short significands (exact products and ties),
    significands of all ones, and zeros, subnormals, infinities and NaN."""
    rng = np.random.default_rng(3)
    n = 1 << 18
    sig = rng.integers(0, 1 << 52, (4, 2, n), dtype=np.uint64)
    sig[1] &= np.uint64(0xffffffe000000)
    sig[2] = (np.uint64(1) << np.uint64(52)) - 1 - (sig[2] & np.uint64(3))
    sig[3, 0] &= np.uint64(0xf000000000000)
    ea = rng.integers(1, 2047, (4, n))
    eb = np.clip(rng.choice([1023, 2046 + 1023 - 1, 1, 1024 + 1023], (4, n))
                 + rng.integers(-3, 4, (4, n))
                 - np.where(rng.random((4, n)) < 0.8, ea - 1023, 0), 1, 2046)
    e = np.stack([ea, eb], axis=1).astype("uint64") << np.uint64(52)
    sign = rng.integers(0, 2, (4, 2, n), dtype=np.uint64) << np.uint64(63)
    x = (sig | e | sign).view("float64")
    special = np.array([0.0, -0.0, 1.0, -1.5, 5e-324, -1e-310, np.inf,
                        -np.inf, np.nan, np.finfo(float).max, 2.0 ** -1022])
    sa, sb = np.meshgrid(special, special)
    return (np.concatenate([x[:, 0].ravel(), sa.ravel()]),
            np.concatenate([x[:, 1].ravel(), sb.ravel()]))


def test_products_are_the_fp64_products():
    from solvcon_gb300._lib import check, lib, ptr
    a, b = _pairs()
    p = np.empty_like(a)
    check(lib.scg_product_check(ptr(a), ptr(b), ptr(p), a.size))
    with np.errstate(all="ignore"):
        want = a * b
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(p), nan)
    np.testing.assert_array_equal(p[~nan].view(np.int64),
                                  want[~nan].view(np.int64))


# A tube of 60,001 points, the smallest that takes the products from the integer
# pipe, and one of 59,999: a point's values after three steps depend on at most
# the seven points on either side.
@pytest.mark.parametrize("alpha", [1, 2])
def test_large_tube_equals_small(alpha):
    import solvcon_gb300.onedim as od
    rng = np.random.default_rng(1)
    big = 60001
    x = np.cumsum(rng.uniform(0.9, 1.1, big)) / big
    so0 = rng.uniform(0.9, 1.1, (big, 3)) * [1.0, 0.2, 2.5]
    so0[big // 3:big // 2, 1] = 0.0
    gamma = rng.uniform(1.2, 1.6, big)
    out = {}
    for n in (big, big - 2):
        core = od.Euler1DCore(n, 0.3 / big)
        core.coord[...], core.gamma[...] = x[:n], gamma[:n]
        core.so0[...], core.so1[...] = so0[:n], 0.0
        core.setup_march()
        getattr(core, "march_alpha%d" % alpha)(3)
        out[n] = [np.array(getattr(core, k)[...])[:big - 16]
                  for k in ("so0", "so1", "cfl")]
    for got, want in zip(out[big], out[big - 2]):
        np.testing.assert_array_equal(got, want)
    assert np.isfinite(out[big][0]).all()


# The same for the spacetime grids: 80,001 elements and 80,000, which are
# periodic, so that both ends are left out.
@pytest.mark.parametrize("solver", ["LinearScalarSolver",
                                    "InviscidBurgersSolver"])
@pytest.mark.parametrize("alpha", [1, 2])
def test_large_grid_equals_small(solver, alpha):
    import solvcon_gb300.spacetime as st
    rng = np.random.default_rng(2)
    big = 80001
    x = np.cumsum(rng.uniform(0.5, 1.5, big + 1))
    out = {}
    for n in (big, big - 1):
        core = getattr(st, solver)(st.Grid(x[:n + 1]), 0.2)
        m = core.so0[...].shape[0]
        wave = np.sin(np.arange(m) / 50.0)
        wave[1000:2000] = 0.0
        core.so0[...] = wave[:, None]
        core.so1[...] = np.cos(np.arange(m) / 70.0)[:, None]
        core.setup_march()
        getattr(core, "march_alpha%d" % alpha)(3)
        out[n] = [np.array(getattr(core, k)[...])[20:2 * (big - 20)]
                  for k in ("so0", "so1", "cfl")]
    for got, want in zip(out[big], out[big - 1]):
        np.testing.assert_array_equal(got, want)
    assert np.isfinite(out[big][0]).all()
