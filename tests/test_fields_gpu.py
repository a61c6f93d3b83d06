"""Tables read back from the device: every value of a record field widened to
FP64 exactly, from single values (the end of a pair) to all special ones."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("cells", ["tri_square", "tet_cube"])
def test_tables_come_back_exactly(precision, aligned, cells):
    """FP32-representable values (zeros of both signs, subnormals, infinities
    and NaN among them) written and read through tables that start on and off
    a 16-byte boundary, with an odd number of values in 3D."""
    import solvcon_gb300 as sg
    from solvcon_gb300 import meshgen
    from solvcon_gb300._lib import check, lib, ptr
    from solvcon_gb300.multidim import _ID
    ndim = 2 if cells == "tri_square" else 3
    mesh = meshgen.build_mesh(ndim, *getattr(meshgen, cells)(3, 0.1, 2))
    core = sg.EulerCore(mesh, 1e-3, precision=precision)
    core.init_solution(1.4, 1.0, [0.0] * ndim, 1.0)
    rng = np.random.default_rng(4)
    special = np.array([0.0, -0.0, 1e-45, -1e-40, 1.1754944e-38, 3.4028235e38,
                        np.inf, -np.inf, np.nan], dtype="float32")
    for name in ("so1c", "so1n", "so0t"):
        shape, _ = core._shape(_ID[name])
        size = int(np.prod(shape))
        value = np.exp2(rng.uniform(-126, 127, size)) * rng.choice([-1, 1], size)
        value[:special.size] = special
        value = value.astype("float32").astype("float64")
        start = 0 if aligned else 1
        src, out = np.empty(size + 2), np.empty(size + 2)
        src[start:start + size] = value
        check(lib.scg_euler_set(core.handle, _ID[name], ptr(src[start:]), size))
        check(lib.scg_euler_get(core.handle, _ID[name], ptr(out[start:]), size))
        got = out[start:start + size]
        nan = np.isnan(value)
        np.testing.assert_array_equal(np.isnan(got), nan, name)
        np.testing.assert_array_equal(got[~nan].view(np.int64),
                                      value[~nan].view(np.int64), name)
