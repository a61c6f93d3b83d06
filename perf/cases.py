"""Performance cases of the CESE march, from the smallest solve to the largest.

Each case is one call (or one exchange) of a user's program on a solver that
it has set up: ``prepare`` builds the mesh or grid, the solver and its initial
state, ``run`` advances it and reads the new state back, ``exact`` marches the
same inputs with plain torch in 64 bits.  A pass continues from the state the
last one left, as a time loop does.

The listed cases and what each stands for:

* ``sod_201``: the reference's own 1D example, a 201-point shock tube marched
  to t = 0.2 in 28 steps: launch and latency bound.
* ``tube_20001_fp32``: one served 1D request (1k to 100k points), FP32 state.
* ``tube_2m``: a large FP64 tube.
* ``scalar_1m``: the spacetime scalar solver on a large periodic grid.
* ``channel_1024``: a small supersonic channel of quadrilaterals with inlet,
  outlet and walls, the size of the oblique-shock example's 64 x 16 mesh.
* ``tri_2m``: the benchmark workload, 2,000,000 jittered triangles in FP64.
* ``exchange_tri_500k``: a host program that feeds the state in and takes it
  out around every step, through page-locked tables.
* ``tri_980k_fp32``: the FP32 form of the 2D march.
* ``tet_384k``: the 3D blast, FP64.
* ``tet_1296k_fp32``: the 3D blast, FP32 form.
* ``hex_64k``: a hexahedral mesh in FP64 (cells that are not simplices).
* ``batch_24_fp32``: many meshes of uneven size in one batched FP32 march.

``draw`` spreads over the same solvers: all cell types, precisions, sizes from
a few hundred points or cells up to the listed ones, both limiter exponents.
"""

import math

import numpy as np
import torch

import solvcon_gb300 as sg
from solvcon_gb300 import meshgen
from solvcon_gb300.batch import EulerBatch
from solvcon_gb300.onedim import Euler1DCore
from solvcon_gb300.spacetime import (Grid, InviscidBurgersSolver,
                                     LinearScalarSolver)
from solvcon_gb300.synth import sod_tube_state

GAMMA = 1.4

# Cells per unit of nside^ndim, faces per cell and the time step as a
# fraction of h / (fastest wave), which gives CFL numbers of 0.2 to 0.6 on the
# jittered meshes.
CELLS = {"tri": (2, 2, 3, 0.10), "quad": (2, 1, 4, 0.25),
         "tet": (3, 6, 4, 0.05), "hex": (3, 1, 6, 0.25),
         "prism": (3, 2, 5, 0.08)}

# Floating-point operations of one cell and substep in the reference's
# formulation with each Jacobian product taken as a directional derivative.
FLOPS = {"tri": 1160, "quad": 1550, "tet": 2720, "hex": 4900, "prism": 3900}


def listed():
    return [
        {"name": "sod_201", "kind": "tube", "n": 201, "precision": "fp64",
         "alpha": 2, "steps": 28},
        {"name": "tube_20001_fp32", "kind": "tube", "n": 20001,
         "precision": "fp32", "alpha": 2, "steps": 200},
        {"name": "tube_2m", "kind": "tube", "n": 2000001,
         "precision": "fp64", "alpha": 2, "steps": 32},
        {"name": "scalar_1m", "kind": "scalar", "pde": "linear",
         "ncelm": 1000000, "alpha": 2, "steps": 32},
        {"name": "channel_1024", "kind": "mesh", "cells": "quad",
         "nside": 32, "precision": "fp64", "walls": "channel", "steps": 20},
        {"name": "tri_2m", "kind": "mesh", "cells": "tri", "nside": 1000,
         "precision": "fp64", "walls": "slip", "steps": 2},
        {"name": "exchange_tri_500k", "kind": "exchange", "cells": "tri",
         "nside": 500, "precision": "fp64", "walls": "slip", "steps": 1},
        {"name": "tri_980k_fp32", "kind": "mesh", "cells": "tri",
         "nside": 700, "precision": "fp32", "walls": "slip", "steps": 20},
        {"name": "tet_384k", "kind": "mesh", "cells": "tet", "nside": 40,
         "precision": "fp64", "walls": "slip", "steps": 2},
        {"name": "tet_1296k_fp32", "kind": "mesh", "cells": "tet",
         "nside": 60, "precision": "fp32", "walls": "slip", "steps": 10},
        {"name": "hex_64k", "kind": "mesh", "cells": "hex", "nside": 40,
         "precision": "fp64", "walls": "slip", "steps": 4},
        {"name": "batch_24_fp32", "kind": "batch", "meshes": 24, "lo": 2000,
         "hi": 200000, "precision": "fp32", "steps": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "tube", "scalar", "mesh", "mesh", "mesh",
                       "mesh", "exchange", "batch"])
    if kind == "tube":
        n = _log_int(rng, 50, 1000000) * 2 + 1
        prec = rng.choice(["fp64", "fp32"])
        top = (32 * 2000001 if prec == "fp64" else 400 * 2000001) // n
        return {"kind": kind, "n": n, "precision": prec,
                "alpha": rng.choice([1, 2]),
                "steps": max(1, min(top, rng.randint(20, 200)))}
    if kind == "scalar":
        n = _log_int(rng, 50, 1000000)
        return {"kind": kind, "pde": rng.choice(["linear", "burgers"]),
                "ncelm": n, "alpha": rng.choice([1, 2]),
                "steps": max(1, min(25000000 // n, rng.randint(20, 200)))}
    if kind == "batch":
        return {"kind": kind, "meshes": rng.randint(2, 24),
                "lo": rng.randint(500, 2000),
                "hi": rng.randint(20000, 150000),
                "precision": rng.choice(["fp32", "fp32", "fp32-geom32"]),
                "steps": rng.randint(2, 20)}
    cells = "tri" if kind == "exchange" else rng.choice(
        ["tri", "tri", "quad", "tet", "tet", "hex", "prism"])
    prec = "fp64" if kind == "exchange" else rng.choice(
        ["fp64", "fp64", "fp32", "fp32", "fp32-geom32"])
    ndim, per, nfc, _ = CELLS[cells]
    top = (1500000 if prec == "fp64" else 4000000) // (1 if ndim == 2 else 4)
    n = max(2, int(round((_log_int(rng, 200, top) / per) ** (1.0 / ndim))))
    # The step count that keeps a pass below the largest listed case's.
    most = (3000000 if prec == "fp64" else 20000000) // \
        ((1 if ndim == 2 else 3) * per * n ** ndim)
    steps = 1 if kind == "exchange" else max(1, min(most, rng.randint(1, 10)))
    return {"kind": kind, "cells": cells, "nside": n, "precision": prec,
            "walls": rng.choice(["slip", "channel"]), "steps": steps}


# ---------------------------------------------------------------------------
# Inputs.

def _geometry(cells, nside, seed):
    """Node coordinates, cell types and cell node lists of a jittered unit
    square or cube."""
    if cells == "tri":
        return meshgen.tri_square(nside, 0.2, seed)
    if cells == "quad":
        return meshgen.quad_square(nside, 0.15, seed)
    if cells == "tet":
        return meshgen.tet_cube(nside, 0.15, seed)
    if cells == "hex":
        return meshgen.hex_cube(nside, 0.1, seed)
    return meshgen.prism_slab(nside, nside, 0.1, seed)


def _node_average(x, c):
    n = int(c[0, 0])
    return x[c[:, 1:1 + n]].mean(axis=1)


def _problem(cells, nside, walls, seed, gamma=GAMMA):
    """A mesh and its initial state: four quadrants of random density,
    pressure and velocity in 2D (through a channel: on a supersonic stream),
    the spherical blast in 3D, with a random density and pressure ratio."""
    ndim, _, _, frac = CELLS[cells]
    rng = np.random.Generator(np.random.PCG64(seed))
    x, t, c = _geometry(cells, nside, seed)
    at = _node_average(x, c)
    if ndim == 2:
        rho, p = rng.uniform(0.1, 1.5, (2, 4))
        vel = rng.uniform(-0.8, 0.8, (4, 2))
        if walls == "channel":
            rho, p, vel = 0.75 + rho / 6, 0.75 + p / 6, vel / 8 + [3.0, 0.0]
        q = (at[:, 0] >= 0.5).astype(int) + 2 * (at[:, 1] >= 0.5)
        rho, p, vel = rho[q], p[q], vel[q]
    else:
        inside = np.linalg.norm(at - 0.5, axis=1) < 0.2
        rho = np.where(inside, rng.uniform(0.8, 1.2),
                       rng.uniform(0.1, 0.15))
        p = np.where(inside, rng.uniform(0.8, 1.2), rng.uniform(0.08, 0.12))
        vel = np.zeros((at.shape[0], 3))
        if walls == "channel":
            vel[:, 0] = 1.0
    wave = np.sqrt((vel ** 2).sum(axis=1)) + np.sqrt(gamma * p / rho)
    free = [1.0] + [3.0 if ndim == 2 else 1.0] + [0.0] * (ndim - 1) + [1.0]
    if walls == "channel":  # the inlet's stream
        wave = np.maximum(wave, free[1] + math.sqrt(gamma))
    return {"ndim": ndim, "x": x, "t": t, "c": c,
            "state": meshgen.conserved(rho, vel, p, gamma),
            "dt": float(frac / nside / wave.max()), "gamma": gamma,
            "walls": walls, "inlet": free + [gamma]}


def _core(pb, precision):
    mesh = meshgen.build_mesh(pb["ndim"], pb["x"], pb["t"], pb["c"])
    core = sg.EulerCore(mesh, pb["dt"], precision=precision)
    core.init_solution(pb["gamma"], 1.0, [0.0] * pb["ndim"], 1.0)
    faces = np.array(mesh.bndfcs.ndarray[:, 0])
    if pb["walls"] == "channel":
        at = np.array(mesh.fccnd[0:])[faces, 0]
        core.add_inlet(faces[at < 1e-12], pb["inlet"])
        core.add_nonrefl(faces[at > 1 - 1e-12])
        faces = faces[(at >= 1e-12) & (at <= 1 - 1e-12)]
    core.add_slipwall(faces)
    core.so0n[0:] = pb["state"]
    core.bc_soln()
    core.bc_dsoln()
    return core


def _mesh_problem(case, seed):
    return _problem(case["cells"], case["nside"], case["walls"], seed)


def _batch_sizes(case):
    """Squares' sides of a batch, cell counts spread evenly over the
    logarithm of their range and shuffled, the same for every seed."""
    n = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]),
                           case["meshes"]))
    np.random.Generator(np.random.PCG64(2026)).shuffle(n)
    return [max(2, int(round(math.sqrt(s / 2)))) for s in n]


def _batch_problems(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    gammas = rng.uniform(1.1, 1.67, case["meshes"])
    return [_problem("tri", n, "slip", seed + 1 + k, float(g))
            for k, (n, g) in enumerate(zip(_batch_sizes(case), gammas))]


def _tube(case, seed):
    """A Sod-type tube on [-1, 1]: random states left and right, at rest."""
    return sod_tube_state(case["n"], seed)


def _scalar(case, seed):
    """A smooth periodic profile of random amplitude and phase."""
    rng = np.random.Generator(np.random.PCG64(seed))
    grid = Grid(0.0, 2.0 * np.pi, case["ncelm"])
    x = np.asarray(grid.xcoord)
    amp, ph = rng.uniform(0.5, 1.0), rng.uniform(0.0, 2.0 * np.pi)
    return (grid, amp * np.sin(x + ph), amp * np.cos(x + ph),
            0.8 * 2.0 * np.pi / case["ncelm"] / 2.0)


# ---------------------------------------------------------------------------
# The measured call.

class _Held:
    """A host table as an array that keeps the table's memory alive."""

    def __init__(self, table):
        self.table = table
        self.__array_interface__ = table.array.__array_interface__


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "tube":
        x, so0, dt = _tube(case, seed)
        core = Euler1DCore(case["n"], dt, precision=case["precision"])
        core.coord[...] = x
        core.so0[...] = so0
        core.setup_march()
        st["core"] = core
    elif kind == "scalar":
        grid, u, ux, dt = _scalar(case, seed)
        cls = {"linear": LinearScalarSolver,
               "burgers": InviscidBurgersSolver}[case["pde"]]
        core = cls(grid, dt)
        core.so0[...] = u[:, None]
        core.so1[...] = ux[:, None]
        core.setup_march()
        st["core"] = core
    elif kind == "batch":
        st["cores"] = [_core(pb, case["precision"])
                       for pb in _batch_problems(case, seed)]
        st["batch"] = EulerBatch(st["cores"], block=128, persistent=False)
    else:
        core = _core(_mesh_problem(case, seed), case["precision"])
        st["core"] = core
        if kind == "exchange":
            st["in"] = [core.host_table(n) for n in ("so0n", "so1n")]
            out = [core.host_table(n) for n in ("so0n", "so1n")]
            for t, n in zip(st["in"], ("so0n", "so1n")):
                t.array[...] = getattr(core, n)[...]
            core.deliver(so0n=out[0], so1n=out[1])
            st["out"] = [np.asarray(_Held(t)) for t in out]
        core.sync()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].march(case["steps"])
        return [[c.so0n[0:], c.so1n[0:]] for c in state["cores"]]
    core = state["core"]
    if kind == "tube":
        (core.march_alpha1 if case["alpha"] == 1 else
         core.march_alpha2)(case["steps"])
        return {"so0": core.so0[...], "so1": core.so1[...],
                "cfl": core.cfl[...]}
    if kind == "scalar":
        (core.march_alpha1 if case["alpha"] == 1 else
         core.march_alpha2)(case["steps"])
        return {"so0": core.so0[...], "so1": core.so1[...],
                "cfl": core.cfl[...]}
    if kind == "exchange":
        core.march_from_host(state["in"][0], state["in"][1], case["steps"])
        g = core.ngstcell
        return {"so0n": state["out"][0][g:], "so1n": state["out"][1][g:]}
    core.march(case["steps"])
    return {"so0n": core.so0n[0:], "so1n": core.so1n[0:],
            "cflo": core.cflo[0:]}


def _mesh_size(case):
    ndim, per, nfc, _ = CELLS[case["cells"]]
    return ndim, per * case["nside"] ** ndim, nfc


def _substeps(state_bytes, case):
    """How often a pass has to move its state: every substep when it is
    larger than the 129 MB L2, once when it stays on the chip."""
    return 2 * case["steps"] if state_bytes > 129e6 else 1


def work(case):
    kind = case["kind"]
    b32 = 4 if case.get("precision", "fp64") != "fp64" else 8
    if kind == "tube":
        # Read so0, so1, gamma and the spacing, write so0, so1 and cfl of a
        # point; half the points in either half step.
        size = case["n"] * b32 * (3 + 3 + 1 + 1 + 3 + 3 + 1)
        return {"bytes": size if size <= 129e6 else size * case["steps"],
                "flops": case["n"] * case["steps"] * 200}
    if kind == "scalar":
        size = 2 * case["ncelm"] * 8 * (1 + 1 + 1 + 1 + 1 + 1)
        return {"bytes": size if size <= 129e6 else size * case["steps"],
                "flops": 2 * case["ncelm"] * case["steps"] * 40}
    if kind == "batch":
        n = sum(2 * side ** 2 for side in _batch_sizes(case))
        ndim, nfc, cells = 2, 3, "tri"
    else:
        ndim, n, nfc = _mesh_size(case)
        cells = case["cells"]
    neq = ndim + 2
    # Per cell and substep: read so0, so1 and gamma, the geometry (a volume
    # and a centroid of the cell and of each of its faces' elements, centroid
    # and normal of each sub-face; FP64 unless the geometry is kept in FP32)
    # and the neighbour ids; write so0, so1 and the two CFL numbers.
    sub = {"tri": 6, "quad": 8, "tet": 12, "hex": 24, "prism": 18}[cells]
    bg = 4 if case["precision"] == "fp32-geom32" else 8
    size = n * ((neq + neq * ndim + 1) * b32 +
                ((1 + nfc) * (1 + ndim) + sub * 2 * ndim) * bg +
                (1 + nfc) * 4 + (neq + neq * ndim + 2) * b32)
    if kind == "exchange":
        return {"bytes": size * 2 + 2 * n * neq * (1 + ndim) * 8,
                "flops": n * 2 * FLOPS[cells]}
    return {"bytes": size * _substeps(size, case),
            "flops": n * 2 * case["steps"] * FLOPS[cells]}


# ---------------------------------------------------------------------------
# The same march in plain torch, 64 bits.

_FACES = {
    "tri": ((0, 1), (1, 2), (2, 0)),
    "quad": ((0, 1), (1, 2), (2, 3), (3, 0)),
    "tet": ((0, 2, 1), (0, 1, 3), (0, 3, 2), (1, 2, 3)),
    "hex": ((0, 3, 2, 1), (1, 2, 6, 5), (4, 5, 6, 7), (0, 4, 7, 3),
            (0, 1, 5, 4), (2, 3, 7, 6)),
    "prism": ((0, 1, 2), (3, 5, 4), (0, 3, 4, 1), (0, 2, 5, 3),
              (1, 4, 5, 2)),
}
# Faces of each fundamental gradient element.
_ELEMS = {
    "tri": ((0, 1), (1, 2), (2, 0)),
    "quad": ((0, 1), (1, 2), (2, 3), (3, 0)),
    "tet": ((2, 0, 1), (1, 0, 3), (3, 0, 2), (1, 3, 2)),
    "hex": ((1, 2, 4), (5, 2, 1), (3, 2, 5), (4, 2, 3), (4, 0, 1),
            (1, 0, 5), (5, 0, 3), (3, 0, 4)),
    "prism": ((4, 1, 3), (2, 1, 4), (3, 1, 2), (3, 0, 4), (4, 0, 2),
              (2, 0, 3)),
}


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


class _Mesh:
    """Connectivity and conservation-element geometry of a single-type mesh,
    [cell, face, ...] tables; boundary faces get a ghost number past the
    cells."""

    def __init__(self, pb, cells):
        dev = _device()
        nd = pb["ndim"]
        faces = _FACES[cells]
        conn = pb["c"][:, 1:1 + int(pb["c"][0, 0])].astype(np.int64)
        nc, nf = conn.shape[0], len(faces)
        x = torch.from_numpy(pb["x"]).to(dev)
        conn = torch.from_numpy(conn).to(dev)
        # Neighbours: equal node sets, two by two.
        key = []
        for f in faces:
            nodes = conn[:, list(f)].sort(dim=1).values
            k = nodes[:, 0]
            for j in range(1, 3 if nd == 3 else 2):
                k = k * pb["x"].shape[0] + nodes[:, j]
            key.append(k)
        key = torch.stack(key, 1).reshape(-1)
        order = torch.argsort(key, stable=True)
        same = key[order][1:] == key[order][:-1]
        first, second = order[:-1][same], order[1:][same]
        nbr = torch.full((nc * nf,), -1, dtype=torch.int64, device=dev)
        nbr[first] = second // nf
        nbr[second] = first // nf
        bnd = (nbr < 0).nonzero().flatten()
        nbr[bnd] = nc + torch.arange(bnd.numel(), device=dev)
        self.nbr = nbr.reshape(nc, nf)
        self.inner = bnd // nf
        self.nc, self.nf, self.nd = nc, nf, nd
        # Face centroids, area vectors; cell centroids.
        avg = x[conn].mean(1)
        cen, area, pts = [], [], []
        for f in faces:
            p = x[conn[:, list(f)]]
            pts.append(p)
            if nd == 2:
                cen.append(p.mean(1))
                e = p[:, 1] - p[:, 0]
                area.append(torch.stack([e[:, 1], -e[:, 0]], 1))
            else:
                m = p.mean(1)
                q = p.roll(-1, 1)
                tri = _cross(p - m[:, None], q - m[:, None])
                w = tri.norm(dim=-1, keepdim=True)
                cen.append(((m[:, None] + p + q) / 3 * w).sum(1) / w.sum(1))
                area.append(tri.sum(1) / 2)
        cen, area = torch.stack(cen, 1), torch.stack(area, 1)
        vob = ((avg[:, None] - cen) * area).sum(-1).abs()[..., None]
        ctr = ((cen + (avg[:, None] - cen) / (nd + 1)) * vob).sum(1) / \
            vob.sum(1)
        out = ((cen - ctr[:, None]) * area).sum(-1).sign()[..., None]
        unit = area * out / area.norm(dim=-1, keepdim=True)
        self.normal = unit.reshape(-1, nd)[bnd]
        self.where = cen.reshape(-1, nd)[bnd]
        off = ((self.where - ctr[self.inner]) * self.normal).sum(-1)
        ghost = ctr[self.inner] + 2 * off[:, None] * self.normal
        allctr = torch.cat([ctr, ghost])
        ce = allctr[self.nbr]  # the neighbours' cell centroids
        # Basic elements, and the moments of their far sub-faces.
        bvol, bcen, subx, subn = [], [], [], []
        for k in range(nf):
            p, e = pts[k], ce[:, k]
            if nd == 2:
                a, b = p[:, 0], p[:, 1]

                def tri_area(c, a=a, b=b):
                    u, v = a - c, b - c
                    return u[:, 0] * v[:, 1] - u[:, 1] * v[:, 0]

                vi = (tri_area(ctr).abs() / 2)[:, None]
                cr = tri_area(e)
                ve = (cr.abs() / 2)[:, None]
                mom = (a + b + ctr) / 3 * vi + (a + b + e) / 3 * ve
                s = torch.where(cr > 0, 1.0, -1.0)[:, None].to(x.dtype)
                bvol.append(vi + ve)
                subx.append(torch.stack([(e + a) / 2, (e + b) / 2], 1))
                subn.append(torch.stack(
                    [torch.stack([-(e - a)[:, 1], (e - a)[:, 0]], 1) * s,
                     torch.stack([-(b - e)[:, 1], (b - e)[:, 0]], 1) * s],
                    1))
            else:
                pf = cen[:, k]
                q = p.roll(-1, 1)
                tri = _cross(p - pf[:, None], q - pf[:, None])
                vi = ((tri * (ctr - pf)[:, None]).sum(-1).abs() /
                      6)[..., None]
                ve = ((tri * (e - pf)[:, None]).sum(-1).abs() / 6)[..., None]
                base = p + q + pf[:, None]
                mom = ((base + ctr[:, None]) / 4 * vi +
                       (base + e[:, None]) / 4 * ve).sum(1)
                bvol.append((vi + ve).sum(1))
                subx.append((e[:, None] + p + q) / 3)
                n = _cross(p - e[:, None], q - e[:, None]) / 2
                subn.append(n * out[:, k, None])  # outward
            bcen.append(mom / bvol[-1])
        self.bvol = torch.stack(bvol, 1)  # [cell, face, 1]
        self.bcen = torch.stack(bcen, 1)
        self.vol = self.bvol.sum(1)
        self.cce = (self.bcen * self.bvol).sum(1) / self.vol
        self.far = torch.cat([self.cce, ghost])[self.nbr]
        self.subx = [s - self.far[:, k, None] for k, s in enumerate(subx)]
        self.subn = subn
        self.dist = (self.bcen - self.cce[:, None]).norm(dim=-1).amin(1)


def _flux(u, ga):
    """Euler flux [row, eq, dim] and its Jacobian's products' ingredients."""
    rho, m, en = u[:, :1], u[:, 1:-1], u[:, -1:]
    v = m / rho
    p = (ga - 1) * (en - 0.5 * (m * v).sum(-1, keepdim=True))
    return rho, m, en, v, p


def _flux_of(u, ga):
    rho, m, en, v, p = _flux(u, ga)
    eye = torch.eye(m.shape[1], dtype=u.dtype, device=u.device)
    mid = m[:, :, None] * v[:, None, :] + p[:, :, None] * eye
    return torch.cat([m[:, None], mid, ((en + p) * v)[:, None]], 1)


def _jvp(u, w, ga):
    """Directional derivative of the flux at u along w [row, eq, k]:
    [row, eq, dim, k]."""
    rho, m, en, v, p = _flux(u, ga)
    w0, wm, we = w[:, :1], w[:, 1:-1], w[:, -1:]
    dv = (wm - v[..., None] * w0) / rho[..., None]
    dp = (ga - 1) * (we - (v[..., None] * wm).sum(1, keepdim=True) +
                     0.5 * (v * v).sum(-1)[:, None, None] * w0)
    eye = torch.eye(m.shape[1], dtype=u.dtype, device=u.device)
    mid = wm[:, :, None] * v[:, None, :, None] + \
        m[:, :, None, None] * dv[:, None] + \
        dp[:, None] * eye[None, :, :, None]
    top = wm[:, None]
    end = (we + dp) * v[..., None] + (en + p)[..., None] * dv
    return torch.cat([top, mid, end[:, None]], 1)


def _march_mesh(pb, cells, steps):
    """(so0n, so1n, cflo) of the body cells after `steps` steps."""
    g = _Mesh(pb, cells)
    dev, nd, nc = _device(), g.nd, g.nc
    ga, dt = pb["gamma"], pb["dt"]
    neq = nd + 2
    nrm = g.normal
    inlet = torch.zeros(g.inner.numel(), dtype=torch.bool, device=dev)
    free = torch.zeros_like(inlet)
    if pb["walls"] == "channel":
        inlet = g.where[:, 0] < 1e-12
        free = g.where[:, 0] > 1 - 1e-12
    rho, p = pb["inlet"][0], pb["inlet"][1 + nd]
    vel = torch.tensor(pb["inlet"][1:1 + nd], dtype=torch.float64)
    feed = torch.cat([torch.tensor([rho], dtype=torch.float64), rho * vel,
                      (p / (ga - 1) + 0.5 * rho * (vel * vel).sum())[None]])
    feed = feed.to(dev)
    refl = torch.eye(nd, dtype=torch.float64, device=dev) - \
        2 * nrm[:, :, None] * nrm[:, None, :]
    proj = torch.eye(nd, dtype=torch.float64, device=dev) - \
        nrm[:, :, None] * nrm[:, None, :]

    def bc0(u):
        b = u[g.inner]
        wall = b.clone()
        wall[:, 1:-1] = (refl @ b[:, 1:-1, None])[..., 0]
        return torch.where(inlet[:, None], feed,
                           torch.where(free[:, None], b, wall))

    def bc1(w):
        b = w[g.inner]
        wall = b @ refl
        wall[:, 1:-1] = refl @ wall[:, 1:-1]
        zero = torch.zeros_like(b)
        return torch.where(inlet[:, None, None], zero,
                           torch.where(free[:, None, None], b @ proj, wall))

    u = torch.from_numpy(pb["state"]).to(dev)
    w = torch.zeros((nc, neq, nd), dtype=torch.float64, device=dev)
    u, w = torch.cat([u, bc0(u)]), torch.cat([w, bc1(w)])
    ne = len(_ELEMS[cells])
    cflo = None
    for _ in range(2 * steps):
        j = _jvp(u, w, ga)  # [row, eq, dim, along]
        t = -torch.diagonal(j, dim1=2, dim2=3).sum(-1)
        f = _flux_of(u, ga) + 0.25 * dt * _jvp(u, t[..., None], ga)[..., 0]
        acc = torch.zeros((nc, neq), dtype=torch.float64, device=dev)
        for k in range(g.nf):
            n = g.nbr[:, k]
            dx = (g.bcen - g.far)[:, k]
            acc += g.bvol[:, k] * (u[n] + (w[n] * dx[:, None]).sum(-1))
            sn = g.subn[k]
            acc -= 0.5 * dt * (f[n] * sn.sum(1)[:, None]).sum(-1)
            mom = (g.subx[k][:, :, None] * sn[..., None]).sum(1)
            acc -= 0.5 * dt * (j[n] * mom[:, None]).sum((-1, -2))
        un = acc / g.vol
        gh0, gh1 = bc0(un), bc1(w)
        rho, m, en, v, _ = _flux(un, ga)
        ke = 0.5 * (m * m).sum(-1, keepdim=True) / rho
        p = (ga - 1) * (en - ke)
        p = (p + p.abs()) / 2
        wave = torch.sqrt(ga * p / rho) + m.norm(dim=-1, keepdim=True) / rho
        cflo = (0.5 * dt * wave)[:, 0] / g.dist
        cflc = (cflo - 1) * (p[:, 0] / (p[:, 0] + 1e-60)) + 1
        un = torch.cat([un[:, :-1], p / (ga - 1) + ke], 1)
        tau = cflc.abs()
        gp = g.bcen + tau[:, None, None] * (g.far - g.bcen)
        dst = gp - gp.mean(1, keepdim=True)
        el = torch.tensor(_ELEMS[cells], device=dev)
        mat = dst[:, el]  # [cell, element, face, dim]
        vob = _det(mat)
        shift = (mat.sum(2) / (nd + 1) * vob[..., None]).sum(1) / \
            vob.sum(1)[:, None]
        idis = dst - shift[:, None]
        jdis = gp - g.far + g.cce[:, None] - \
            (gp.mean(1) + shift)[:, None]
        du = torch.stack(
            [u[g.nbr[:, k]] + 0.5 * dt * t[g.nbr[:, k]] - un +
             (w[g.nbr[:, k]] * jdis[:, k, None]).sum(-1)
             for k in range(g.nf)], 1)
        inv = _inverse(idis[:, el])
        grad = [(inv[:, e, None] * du[:, el[e]].transpose(1, 2)
                 [:, :, None]).sum(-1) for e in range(ne)]  # [cell, eq, dim]
        wgt = [1 / torch.sqrt((q * q).sum(-1) + 1e-200) for q in grad]
        tot = sum(wgt)
        wgt = [q / tot - 1.0 / ne for q in wgt]
        hi = torch.stack(wgt).amax(0).clamp(min=0)
        lo = torch.stack(wgt).amin(0).clamp(max=0)
        sm = torch.minimum((1 - 1.0 / ne) / (hi + 1e-200),
                           -(1.0 / ne) / (lo - 1e-200))
        sm = torch.minimum(sm, (3.0 / tau)[:, None])
        wn = sum((1.0 / ne + sm * q)[..., None] * d
                 for q, d in zip(wgt, grad))
        u, w = torch.cat([un, gh0]), torch.cat([wn, gh1])
    return u[:nc], w[:nc], cflo


def _det(a):
    if a.shape[-1] == 2:
        return a[..., 0, 0] * a[..., 1, 1] - a[..., 0, 1] * a[..., 1, 0]
    return (a[..., 0, :] * _cross(a[..., 1, :], a[..., 2, :])).sum(-1)


def _inverse(a):
    """Inverse of the last two dimensions (2 x 2 or 3 x 3)."""
    if a.shape[-1] == 2:
        adj = torch.stack([torch.stack([a[..., 1, 1], -a[..., 0, 1]], -1),
                           torch.stack([-a[..., 1, 0], a[..., 0, 0]], -1)],
                          -2)
    else:
        r0, r1, r2 = a[..., 0, :], a[..., 1, :], a[..., 2, :]
        adj = torch.stack([_cross(r1, r2), _cross(r2, r0), _cross(r0, r1)],
                          -1)
    return adj / _det(a)[..., None, None]


def _march_tube(case, seed):
    """so0, so1, cfl of the whole tube after case["steps"] steps."""
    x, so0, dt = _tube(case, seed)
    dev = _device()
    n = case["n"]
    x = torch.from_numpy(x).to(dev)
    u = torch.from_numpy(so0).to(dev)
    w = torch.zeros_like(u)
    cfl = torch.zeros(n, dtype=torch.float64, device=dev)
    ga, tiny = GAMMA, 1e-100

    def half(odd):
        a = 1 if odd else 2
        stop = n - 2 - (0 if odd else 1)
        i = torch.arange(a, stop + 2, 2, device=dev)
        if i[-1] > n - 2:
            i = i[:-1]
        xl, xc, xr = x[i - 1], x[i], x[i + 1]
        ctr = (xl + xr) / 2
        ui, wi = u[i], w[i]
        f = _flux_of(ui, ga)[..., 0]
        t = -_jvp(ui, wi[..., None], ga)[..., 0, 0]
        ft = _jvp(ui, t[..., None], ga)[..., 0, 0]
        off = (xc - ctr)[:, None]
        up = ui + off * wi + dt / 2 * t
        tf = dt / 2 * (f - off * t + dt / 4 * ft)
        ll = (xr - xc)[:, None] * (ui + ((xc + xr) / 2 - ctr)[:, None] * wi)
        lr = (xc - xl)[:, None] * (ui + ((xc + xl) / 2 - ctr)[:, None] * wi)
        new = (ll[:-1] + tf[:-1] + lr[1:] - tf[1:]) / \
            (x[i[1:]] - x[i[:-1]])[:, None]
        k = i[:-1]
        rho, m, en, v, p = _flux(u[k], ga)
        p = (p + p.abs()) / 2
        cfl[k] = dt / 2 * (torch.sqrt(ga * p / rho) + v.abs())[:, 0] / \
            torch.minimum(x[k + 1] - x[k], x[k] - x[k - 1])
        u[k + 1] = new
        dn = (new - up[:-1]) / (x[k + 1] - x[k])[:, None]
        dp = (up[1:] - new) / (x[k + 2] - x[k + 1])[:, None]
        an, ap = dn.abs() ** case["alpha"], dp.abs() ** case["alpha"]
        w[k + 1] = (ap * dn + an * dp) / (ap + an + tiny)

    for _ in range(case["steps"]):
        half(False)
        for s in (u, w):
            s[1] = s[2]
            s[n - 2] = s[n - 3]
        half(True)
    return u, w, cfl


def _march_scalar(case, seed):
    grid, u, ux, dt = _scalar(case, seed)
    dev = _device()
    x = torch.from_numpy(np.array(grid.xcoord)).to(dev)
    u, w = torch.from_numpy(u).to(dev), torch.from_numpy(ux).to(dev)
    cfl = torch.zeros_like(u)
    n, lin = case["ncelm"], case["pde"] == "linear"

    def number(k):
        speed = torch.ones_like(u[k]) if lin else u[k].abs()
        return dt / 2 * speed / torch.minimum(x[k] - x[k - 1],
                                              x[k + 1] - x[k])

    last = 2 * n + 1
    k = torch.arange(2, 2 * n + 3, 2, device=dev)
    cfl[k] = number(k)
    for _ in range(case["steps"]):
        for odd in (0, 1):
            c = torch.arange(-odd, n, device=dev)
            i = 2 + 2 * torch.arange(-odd, n + 1, device=dev) + odd
            xl, xc, xr = x[i - 1], x[i], x[i + 1]
            ctr = (xl + xr) / 2
            ui, wi, off = u[i], w[i], xc - ctr
            xn = (xc - xl) * (ui + ((xl + xc) / 2 - ctr) * wi)
            xp = (xr - xc) * (ui + ((xr + xc) / 2 - ctr) * wi)
            if lin:
                tp = dt / 2 * (ui + off * wi - dt / 4 * wi)
            else:
                tp = dt / 2 * (0.5 * ui * ui + off * ui * wi -
                               dt / 4 * ui * ui * wi)
            nxt = ui + off * wi - dt / 2 * wi
            top = 3 + 2 * c + odd
            new = (xp[:-1] + tp[:-1] + xn[1:] - tp[1:]) / \
                (x[top + 1] - x[top - 1])
            dn = (new - nxt[:-1]) / (xr - xc)[:-1]
            dp = (nxt[1:] - new) / (xc - xl)[1:]
            an, ap = dn.abs() ** case["alpha"], dp.abs() ** case["alpha"]
            u[top] = new
            w[top] = (ap * dn + an * dp) / (ap + an + 2.0 ** -1022)
            if not odd:
                for s in (u, w):
                    inner = s[3].clone()
                    s[1] = s[last]
                    s[last + 2] = inner
                ends = torch.tensor([1, last + 2], device=dev)
                cfl[ends] = number(ends)
            cfl[top] = number(top)
    return u, w, cfl


def exact(case, seed):
    kind = case["kind"]
    if kind == "tube":
        u, w, c = _march_tube(case, seed)
        return {"so0": u, "so1": w, "cfl": c}
    if kind == "scalar":
        u, w, c = _march_scalar(case, seed)
        return {"so0": u[:, None], "so1": w[:, None], "cfl": c}
    if kind == "batch":
        return [list(_march_mesh(pb, "tri", case["steps"])[:2])
                for pb in _batch_problems(case, seed)]
    u, w, c = _march_mesh(_mesh_problem(case, seed), case["cells"],
                          case["steps"])
    out = {"so0n": u, "so1n": w}
    if kind == "mesh":
        out["cflo"] = c
    return out
