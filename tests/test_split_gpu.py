"""Small FP64 meshes, marched with several lanes per cell, against the batched
march of the same mesh, which takes one lane per cell: the same bits."""

import numpy as np
import pytest

from _util import fixture_mesh

pytestmark = pytest.mark.gpu


def _core(mesh, ndim):
    import solvcon_gb300 as sg
    from solvcon_gb300 import meshgen
    core = sg.EulerCore(mesh, 1e-3)
    core.init_solution(1.4, 1.0, [0.3] * ndim, 1.0)
    clcnd = np.array(mesh.clcnd.ndarray)[mesh.ngstcell:]
    core.so0n[0:] = meshgen.quadrant_state(clcnd[:, :2], 3) if ndim == 2 \
        else meshgen.blast_state(clcnd, radius=0.4)
    faces = [int(f) for f in mesh.bndfcs.ndarray[:, 0]]
    core.add_slipwall(faces[0::3])
    core.add_nonrefl(faces[1::3])  # every third face keeps its stale ghost
    core.bc_soln()
    core.bc_dsoln()
    return core


# Every cell type, both mixtures, one cell, cells that fill a warp's groups
# and ones that leave some empty, and the last mesh with several lanes per cell
# and the first with one (12,800 cells in 2D, 5,200 in 3D).
@pytest.mark.parametrize("name,args", [
    ("quad1", None), ("mixed", None), ("tet1", None), ("hex1", None),
    ("pyr1", None), ("prism1", None), ("tri3", None),
    ("tri_square", (2, 0.2, 4)), ("tri_square", (5, 0.2, 4)),
    ("tri_square", (80, 0.2, 4)), ("tri_square", (81, 0.2, 4)),
    ("quad_square", (11, 0.15, 5)), ("quad_square", (113, 0.15, 5)),
    ("tet_cube", (3, 0.15, 6)), ("tet_cube", (9, 0.15, 6)),
    ("tet_cube", (10, 0.15, 6)), ("hex_cube", (5, 0.1, 7)),
    ("hex_cube", (17, 0.1, 7)), ("prism_slab", (7, 3, 0.1, 8))])
def test_lanes_per_cell_leave_the_bits(name, args):
    from solvcon_gb300 import meshgen
    from solvcon_gb300.batch import EulerBatch
    if args is None:
        mesh = fixture_mesh(name)
        ndim = mesh.ndim
    else:
        ndim = 2 if name in ("tri_square", "quad_square") else 3
        mesh = meshgen.build_mesh(ndim, *getattr(meshgen, name)(*args))
    a, b = _core(mesh, ndim), _core(mesh, ndim)
    a.march(3)
    EulerBatch([b], block=128).march(3)
    for table in ("so0c", "so0n", "so0t", "so1c", "so1n", "cflo", "cflc"):
        np.testing.assert_array_equal(getattr(a, table).ndarray,
                                      getattr(b, table).ndarray, table)
    np.testing.assert_array_equal(a.limiter_mask(), b.limiter_mask())
    assert np.isfinite(a.so0n[0:]).all()
