"""The FP64 gradient elements' weights: in integers over the range of sigma0
that the fixed point takes, by FP64 operations beyond it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS = [("tri_square", (6, 0.2, 4)), ("quad_square", (6, 0.15, 5)),
         ("tet_cube", (2, 0.15, 6)), ("hex_cube", (3, 0.1, 7)),
         ("prism_slab", (3, 2, 0.1, 8))]


def _march(cells, args, sigma0, scale=1.0, steps=2):
    import solvcon_gb300 as sg
    from solvcon_gb300 import meshgen
    ndim = 2 if cells in ("tri_square", "quad_square") else 3
    mesh = meshgen.build_mesh(ndim, *getattr(meshgen, cells)(*args))
    core = sg.EulerCore(mesh, 1e-3)
    core.sigma0 = sigma0
    core.init_solution(1.4, 1.0, [0.0] * ndim, 1.0)
    clcnd = np.array(mesh.clcnd.ndarray)[mesh.ngstcell:]
    state = meshgen.quadrant_state(clcnd[:, :2], 3) if ndim == 2 \
        else meshgen.blast_state(clcnd, radius=0.4)
    # Density, momentum and energy scaled alike: the same flow.
    core.so0n[0:] = state * scale
    core.add_slipwall([int(f) for f in mesh.bndfcs.ndarray[:, 0]])
    core.bc_soln()
    core.bc_dsoln()
    core.march(steps)
    return (np.array(core.so0n[0:]), np.array(core.so1n[0:]),
            np.array(core.limiter_mask()))


# (N - 1) |cfl| / sigma0 within 2^[-400, 400) (|cfl| is at least the smallest of
# these marches', 1e-3): sigma0 = 1e115 and 1e-115 are within, 1e125 and 1e-125
# beyond.  At the one end every weight is capped, at the other none differs
# from 1/N beyond 1e-100.
@pytest.mark.parametrize("cells,args", CELLS)
@pytest.mark.parametrize("inside,beyond", [(1e115, 1e125), (1e-115, 1e-125)])
def test_sigma0_beyond_the_fixed_point(cells, args, inside, beyond):
    """The weights of both routes differ by rounding, 2^-52 of their sum; a
    gradient by that times the elements' spread, below 1e-12 of the largest."""
    got, want = (_march(cells, args, s) for s in (inside, beyond))
    for g, w in zip(got[:2], want[:2]):
        np.testing.assert_allclose(g, w, rtol=0, atol=1e-11 * abs(w).max())
    assert np.isfinite(got[1]).all()


@pytest.mark.parametrize("cells,args", CELLS)
def test_flow_of_any_magnitude(cells, args):
    """A power of two in all conserved variables scales the results by it,
    while squared gradients stay far above 1e-200."""
    got = _march(cells, args, 3.0, 2.0 ** 40)
    want = _march(cells, args, 3.0)
    for g, w in zip(got[:2], want[:2]):
        np.testing.assert_allclose(g * 2.0 ** -40, w, rtol=0,
                                   atol=1e-11 * abs(w).max())
