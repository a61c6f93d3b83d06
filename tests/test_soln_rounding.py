"""Rounding of the FP64 calc_soln (soln64 and soln64_eq of euler_fp64.cuh,
compiled for the host) against the same sums in exact arithmetic.

A cell's new state is the neighbours' values times their volumes, summed, plus
many smaller flux and gradient terms.  Where the volumes' terms are added last,
only they and the final product round at the sum's magnitude: NFC + 1 roundings
of at most 2^-53 of it.  The smaller terms here are below 2^-12 of the volumes',
so that their own roundings, ND (ND + 2) a face, add less than
NFC ND (ND + 2) 2^-11 of one more (0.05; 0.1 is allowed)."""

import ctypes
from fractions import Fraction

import numpy as np
import pytest

from _device_host import library

CODE = r"""
using namespace scg::dev;
template <int CT>
static void soln(double const * cur, double const * geo, int32_t const * nbr, double * out, double * eq)
{
    MarchArgs<double, double> a{};
    a.cur = cur;
    a.geo = geo;
    a.nbr = nbr;
    a.ncell = 1;
    a.npl = Dim<CellT<CT>::ND>::KC + CellT<CT>::NFC * Geo<CellT<CT>::ND, double>::KF;
    soln64<CT, true>(a, 0, out);
    for (int q = 0; q < CellT<CT>::ND + 2; ++q)
        eq[q] = soln64_eq<CT>(a, 0, q);
}
extern "C" void soln(int ct, double const * cur, double const * geo, int32_t const * nbr, double * out, double * eq)
{
    switch (ct)
    {
    case 3: soln<3>(cur, geo, nbr, out, eq); break;
    case 4: soln<4>(cur, geo, nbr, out, eq); break;
    case 5: soln<5>(cur, geo, nbr, out, eq); break;
    case 6: soln<6>(cur, geo, nbr, out, eq); break;
    case 7: soln<7>(cur, geo, nbr, out, eq); break;
    default: soln<8>(cur, geo, nbr, out, eq); break;
    }
}
"""

# Faces, and dimensions, of the cell types.
CELLS = {"quadrilateral": (3, 4, 2), "triangle": (4, 3, 2),
         "hexahedron": (5, 6, 3), "tetrahedron": (6, 4, 3),
         "prism": (7, 5, 3), "pyramid": (8, 5, 3)}
TILE = 32


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return library(tmp_path_factory.mktemp("soln"), CODE,
                   ("divide.cuh", "euler_device.cuh", "euler_fp64.cuh"))


def _sym(k, d, nd):
    a, b = min(k, d), max(k, d)
    return a * nd - a * (a - 1) // 2 + b - a


def _sums(nfc, nd, rec, face, ivol):
    """Each equation's sum and result, exactly."""
    neq = nd + 2
    ns = nd * (nd + 1) // 2
    op = 2 * neq + neq * nd
    am, ae = nd, nd + ns
    bm = ae + nd
    be = bm + ns * nd
    frac = np.vectorize(Fraction)
    rec, face = frac(rec), frac(face)
    out = []
    for q in range(neq):
        s = Fraction(0)
        for f in range(nfc):
            r, g = rec[f], face[f]
            c = r[op:]
            grad = r[2 * neq:op].reshape(neq, nd)
            s += g[0] * r[q]
            for d in range(nd):
                a = c[d] if q == 0 else (c[ae + d] if q == neq - 1
                                         else c[am + _sym(q - 1, d, nd)])
                s += g[1 + d] * grad[q, d] - g[1 + nd + d] * a
                for e in range(nd):
                    b = grad[1 + d, e] if q == 0 else (
                        c[be + d * nd + e] if q == neq - 1
                        else c[bm + _sym(q - 1, d, nd) * nd + e])
                    s -= g[1 + 2 * nd + e * nd + d] * b
        out.append(s * Fraction(ivol))
    return out


@pytest.mark.parametrize("name", sorted(CELLS))
def test_sums_round_as_often_as_they_have_faces(lib, name):
    ct, nfc, nd = CELLS[name]
    neq = nd + 2
    rs = 36 if nd == 2 else 64
    kf = 1 + 5 * nd + nd * nd
    rng = np.random.Generator(np.random.PCG64(ct))
    vp = ctypes.c_void_p
    worst = 0.0
    for _ in range(400):
        rec = np.zeros((nfc, rs))
        rec[:, :neq] = 1.0 + 0.01 * rng.random((nfc, neq))
        rec[:, 2 * neq:] = rng.uniform(-1, 1, (nfc, rs - 2 * neq)) * 2.0 ** -12
        face = np.zeros((nfc, kf))
        face[:, 0] = (1.0 + 0.01 * rng.random(nfc)) / nfc
        face[:, 1:1 + 2 * nd + nd * nd] = rng.uniform(
            -1, 1, (nfc, 2 * nd + nd * nd)) / nfc
        ivol = 1.0 + 0.01 * rng.random()
        geo = np.zeros((2 + nfc * kf, TILE))
        geo[0, 0] = ivol
        geo[2:, 0] = face.ravel()
        nbr = np.arange(nfc, dtype=np.int32)
        got, eq = np.empty(neq), np.empty(neq)
        lib.soln(ct, vp(rec.ctypes.data), vp(geo.ctypes.data),
                 vp(nbr.ctypes.data), vp(got.ctypes.data),
                 vp(eq.ctypes.data))
        np.testing.assert_array_equal(got, eq)
        for q, want in enumerate(_sums(nfc, nd, rec, face, ivol)):
            off = abs(Fraction(float(got[q])) - want) / abs(want) * 2 ** 53
            worst = max(worst, float(off))
    terms = 0 if name != "triangle" else nfc * nd * (nd + 2)
    assert worst <= nfc + 1.1 + terms, worst
