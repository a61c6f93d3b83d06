"""The served solvers' device memory against the HBM budget, in FP64."""

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _server(budget, n=40):
    from solvcon_gb300 import meshgen
    from solvcon_gb300.serving import Server
    srv = Server(hbm_budget=budget, max_chunk=8, precision="fp64")
    x, t, c = meshgen.tri_square(n, 0.2, 1)
    mesh = meshgen.build_mesh(2, x, t, c)
    clcnd = np.asarray(mesh.clcnd.ndarray)[mesh.ngstcell:]
    state = meshgen.quadrant_state(clcnd, 1, 1.4)
    faces = np.asarray(mesh.bndfcs.ndarray[:, 0]).copy()
    srv.add_mesh(0, mesh, state, faces, 1.4, 1e-3)
    return srv, mesh


def _serve(srv, reqs):
    # Every request has arrived by the first tick.
    done = srv.run(reqs, clock=itertools.count(0.0, 1.0).__next__)
    return sorted(r.rid for r in done)


def test_meshes_that_do_not_fit_wait():
    """Room for one solver and a bit: two requests run one after the other."""
    import solvcon_gb300 as sg
    from solvcon_gb300.serving import Request
    srv, mesh = _server(0)
    one = sg.EulerCore(mesh, 1e-3).device_bytes
    for budget, resident in ((2 * one - 1, 1), (2 * one, 2)):
        srv, _ = _server(budget)
        reqs = [Request(k, "2d", 9, 0.0, mesh_key=0) for k in range(2)]
        assert _serve(srv, reqs) == [0, 1]
        assert srv.peak_resident == resident and srv.peak_held <= budget
    srv, _ = _server(one - 1)
    assert _serve(srv, [Request(0, "2d", 9, 0.0, mesh_key=0)]) == []
    assert [r.rid for r in srv.rejected] == [0]


def test_tubes_count_what_they_hold():
    """An FP64 tube's tables: peak of what its core allocates."""
    import gc
    from solvcon_gb300._lib import lib
    from solvcon_gb300.onedim import Euler1DCore
    from solvcon_gb300.serving import Server
    for precision in ("fp64", "fp32"):
        gc.collect()
        lib.scg_device_peak_bytes(1)
        before = lib.scg_device_peak_bytes(0)
        core = Euler1DCore(10001, 1e-4, precision=precision)
        core.so0[...] = 1.0
        core.setup_march()
        np.array(core.so0[...])
        held = lib.scg_device_peak_bytes(0) - before
        assert 0 < held <= Server.tube_bytes(10001, precision)
        del core
