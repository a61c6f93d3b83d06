"""Device memory of a core's set-up."""

import gc

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,args", [("tri_square", (60, 0.2, 4)),
                                        ("quad_square", (60, 0.15, 5)),
                                        ("tet_cube", (12, 0.15, 6)),
                                        ("hex_cube", (20, 0.1, 7))])
def test_records_and_sub_face_tables_are_not_held_at_once(cells, args):
    """While a core is made its buffers hold at most what it keeps, or what it
    keeps without the two record buffers (36 or 64 reals a row and buffer) and
    with the two sub-face tables (24 ndim values a cell each)."""
    import solvcon_gb300 as sg
    from solvcon_gb300 import meshgen
    from solvcon_gb300._lib import lib
    ndim = 2 if cells in ("tri_square", "quad_square") else 3
    mesh = meshgen.build_mesh(ndim, *getattr(meshgen, cells)(*args))
    gc.collect()
    lib.scg_device_peak_bytes(1)
    before = lib.scg_device_peak_bytes(0)
    core = sg.EulerCore(mesh, 1e-3)
    peak = lib.scg_device_peak_bytes(0) - before
    keeps = core.device_bytes
    records = 2 * 8 * (36 if ndim == 2 else 64) * (mesh.ncell + mesh.ngstcell)
    tables = 2 * 8 * 24 * ndim * mesh.ncell
    # The boundary tables and the limiter mask, which device_bytes leaves out.
    slack = 64 * mesh.ngstcell + 2 * mesh.ncell + 4096
    assert peak <= max(keeps, keeps - records + tables) + slack
    del core
    lib.scg_device_peak_bytes(1)
    assert lib.scg_device_peak_bytes(0) == before
