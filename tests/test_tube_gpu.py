"""Whole marches of 1D tubes and spacetime grids in one launch (the points in
the registers of a cluster of blocks) against the same steps taken one method
at a time, at the sizes where threads, warps and blocks of the cluster begin
and end."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _core(n, precision, seed):
    import solvcon_gb300.onedim as od
    from solvcon_gb300.synth import sod_tube_state
    rng = np.random.default_rng(seed)
    x, so0, dt = sod_tube_state(n, seed)
    x[1:-1] += rng.uniform(-0.2, 0.2, n - 2) * (x[1] - x[0])
    so0 *= rng.uniform(0.9, 1.1, (n, 1))
    core = od.Euler1DCore(n, dt, precision=precision)
    core.coord[...] = x
    core.gamma[...] = rng.uniform(1.2, 1.6, n)
    core.so0[...] = so0
    core.so1[...] = 0.0
    core.setup_march()
    return core


# Point pairs (n - 1) / 2 per thread: one thread, a warp less, exactly, and more
# than full, two blocks of one warp, 16 blocks, their second warp, the last
# tube that fits (FP64 4,097, FP32 32,769) and the first that does not.
@pytest.mark.parametrize("precision,sizes", [
    ("fp64", (5, 7, 63, 65, 67, 129, 1025, 1027, 2001, 4097, 4099)),
    ("fp32", (7, 63, 65, 67, 129, 1025, 1027, 4097, 32769, 32771, 400001,
              400003))])
@pytest.mark.parametrize("alpha", [1, 2])
def test_march_equals_its_half_steps(precision, sizes, alpha):
    """march_alpha(3) leaves bit for bit what three times the half-step
    methods leave (they run one launch each, and share its arithmetic)."""
    for n in sizes:
        got, want = _core(n, precision, n), _core(n, precision, n)
        getattr(got, "march_alpha%d" % alpha)(3)
        for _ in range(3):
            getattr(want, "march_half1_alpha%d" % alpha)()
            want.treat_boundary_so0()
            want.treat_boundary_so1()
            getattr(want, "march_half2_alpha%d" % alpha)()
        for name in ("so0", "so1", "cfl"):
            np.testing.assert_array_equal(getattr(got, name)[...],
                                          getattr(want, name)[...],
                                          "%s n=%d" % (name, n))
        assert np.isfinite(got.so0[...]).all()


# Point pairs ncelm + 2: one element, a warp's end, two warps, 16 blocks, their
# second and eighth warp, the last grid that fits (4,094) and the first that
# does not.
@pytest.mark.parametrize("solver", ["LinearScalarSolver",
                                    "InviscidBurgersSolver"])
@pytest.mark.parametrize("alpha", [1, 2])
def test_spacetime_march_equals_its_half_steps(solver, alpha):
    """march_alpha(3) leaves bit for bit what the half-step methods leave."""
    import solvcon_gb300.spacetime as st
    for n in (1, 2, 29, 30, 31, 62, 63, 510, 511, 4094, 4095):
        rng = np.random.default_rng(n)
        grid = st.Grid(np.cumsum(rng.uniform(0.5, 1.5, n + 1)))
        cores = []
        for _ in range(2):
            core = getattr(st, solver)(grid, 0.2)
            x = grid.xcoord
            core.so0[...] = np.sin(x)[:, None]
            core.so1[...] = np.cos(x)[:, None]
            core.setup_march()
            cores.append(core)
        got, want = cores
        getattr(got, "march_alpha%d" % alpha)(3)
        for _ in range(3):
            getattr(want, "march_half1_alpha%d" % alpha)()
            getattr(want, "march_half2_alpha%d" % alpha)()
        for name in ("so0", "so1", "cfl"):
            np.testing.assert_array_equal(getattr(got, name)[...],
                                          getattr(want, name)[...],
                                          "%s ncelm=%d" % (name, n))
        assert np.isfinite(got.so0[...]).all()
