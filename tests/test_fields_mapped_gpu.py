"""Tables exchanged with page-locked host memory, which the device reads and
writes directly: every kind of value, on and off a 16-byte boundary (where a
thread's pair of values moves one by one), an odd number of values in 3D."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("cells", ["tri_square", "tet_cube"])
def test_mapped_tables_come_back_exactly(precision, skip, cells):
    """FP32-representable values, zeros of both signs, subnormals, infinities
    and NaN among them; so0n, whose FP32 rounding residual is kept and added
    back, with finite ones and as numbers (-0 comes back as 0)."""
    import solvcon_gb300 as sg
    from solvcon_gb300 import meshgen
    from solvcon_gb300._lib import check, lib
    from solvcon_gb300.host import HostTable
    from solvcon_gb300.multidim import _ID
    ndim = 2 if cells == "tri_square" else 3
    mesh = meshgen.build_mesh(ndim, *getattr(meshgen, cells)(3, 0.1, 2))
    core = sg.EulerCore(mesh, 1e-3, precision=precision)
    core.init_solution(1.4, 1.0, [0.0] * ndim, 1.0)
    rng = np.random.default_rng(6)
    special = np.array([0.0, -0.0, 1e-45, -1e-40, 1.1754944e-38, 3.4028235e38,
                        np.inf, -np.inf, np.nan], dtype="float32")
    for name in ("so1c", "so1n", "so0t", "so0n"):
        size = int(np.prod(core._shape(_ID[name])[0]))
        src, out = HostTable(size + 2), HostTable(size + 2)
        value = np.exp2(rng.uniform(-126, 127, size)) * rng.choice([-1, 1], size)
        value[:special.size] = special if name != "so0n" else np.where(
            np.isfinite(special), special, 1.0)
        value = value.astype("float32").astype("float64")
        out.array[...] = 7.0
        src.array[skip:skip + size] = value
        check(lib.scg_euler_set(core.handle, _ID[name],
                                ctypes.c_void_p(src.address + 8 * skip), size))
        check(lib.scg_euler_get(core.handle, _ID[name],
                                ctypes.c_void_p(out.address + 8 * skip), size))
        got = out.array[skip:skip + size]
        if name == "so0n":
            np.testing.assert_array_equal(got, value)
        else:
            nan = np.isnan(value)
            np.testing.assert_array_equal(np.isnan(got), nan, name)
            np.testing.assert_array_equal(got[~nan].view(np.int64),
                                          value[~nan].view(np.int64), name)
        # Nothing outside the table.
        assert (out.array[:skip] == 7.0).all()
        assert (out.array[skip + size:] == 7.0).all()
