"""The workloads whose speed is followed: model steps of the sea-ice dynamics,
batched ensembles and the column thermodynamics, through the package's public
classes.

Every dynamics case is the step a host model makes around the kernel
(MEVPDynamics / BBMDynamics): the cell averages of thickness, concentration
(and damage), the wind, the ocean current and the sea-surface height go in
from host arrays, one update runs, the updated cell averages come back to host
arrays.  Cells are 4 km wide (25 km on the sphere), the time step is 120 s and
the mEVP relaxation constants are the library's defaults.

Precision "fp64" returns float64 throughout.  On the "mixed" path the velocity
sub-cycle, the ice-ocean stress and the BBM damage are computed in 32 bits:
these outputs are kept as float32, as a program that writes them to
single-precision files keeps them; thickness and concentration are FP64
fields on either path and are returned as float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nextsimdg_gb300.dynamics import BBMDynamicsKernel, Ensemble, MEVPDynamicsKernel
from nextsimdg_gb300.ice_growth import IceGrowth

DT = 120.0
CELL = 4000.0  # [m]
SUB = 100      # sub-cycle iterations of a model step

MODULE_IN = ("hice", "cice", "uwind", "vwind", "uocean", "vocean", "ssh")
MODULE_OUT = ("hice", "cice", "u", "v", "uiostress", "viostress")
ENSEMBLE_IN = ("hice", "cice", "uwind", "vwind")
ENSEMBLE_OUT = ("hice", "cice", "u", "v")
GROWTH_IN = ("hice", "cice", "hsnow", "tice", "qia", "dqia_dt", "qow", "qio", "sublim", "snowfall", "penSW", "sst",
             "damage")
GROWTH_FIXED = ("tf", "mlbhc")
GROWTH_OUT = ("hice_updated", "cice_updated", "hsnow_updated", "tice_updated", "newice", "qow", "qio", "damage")
GROWTH_DT = 600.0


def _dyn(rheology, mesh, nx, ny, dg, precision):
    return {"kind": "dynamics", "rheology": rheology, "mesh": mesh, "nx": nx, "ny": ny, "dg": dg,
            "precision": precision}


def listed():
    return [
        # a small box with linear advection, as a test or a tutorial runs it: launch latency
        dict(_dyn("mevp", "box", 64, 64, 3, "fp64"), name="box64_dg1_fp64"),
        # the drop-in path (the reference's FP64 arithmetic) on a regular grid
        dict(_dyn("mevp", "box", 256, 256, 6, "fp64"), name="box256_fp64"),
        # the drop-in path on general quadrilaterals (a curvilinear regional grid), odd sizes
        dict(_dyn("mevp", "quads", 201, 143, 6, "fp64"), name="quads201_fp64"),
        # the drop-in path on a lon/lat patch of the sphere (the Arctic grids are of this size)
        dict(_dyn("mevp", "sphere", 154, 121, 6, "fp64"), name="sphere154_fp64"),
        # the small box on the mixed path
        dict(_dyn("mevp", "box", 64, 64, 3, "mixed"), name="box64_dg1_mixed"),
        # the production path on the benchmark grid
        dict(_dyn("mevp", "box", 512, 512, 6, "mixed"), name="box512_mixed"),
        # the production path on general quadrilaterals
        dict(_dyn("mevp", "quads", 384, 320, 6, "mixed"), name="quads384_mixed"),
        # the production path on the sphere, with linear advection
        dict(_dyn("mevp", "sphere", 301, 257, 3, "mixed"), name="sphere301_dg1_mixed"),
        # the brittle rheology, drop-in and production path
        dict(_dyn("bbm", "box", 96, 80, 6, "fp64"), name="bbm96_fp64"),
        dict(_dyn("bbm", "box", 256, 256, 6, "mixed"), name="bbm256_mixed"),
        # an ensemble of uneven domains stepped together
        {"kind": "ensemble", "members": 8, "least": 64, "most": 192, "dg": 6, "name": "ensemble8_mixed"},
        # the column thermodynamics of the same grid as the production path
        {"kind": "growth", "cells": 512 * 512, "name": "ice_growth_512x512"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dynamics"] * 6 + ["ensemble", "growth"])
    if kind == "ensemble":
        return {"kind": "ensemble", "members": rng.randint(2, 8), "least": rng.randint(24, 64),
                "most": rng.randint(65, 180), "dg": rng.choice([1, 3, 6])}
    if kind == "growth":
        return {"kind": "growth", "cells": size(4000, 512 * 512)}
    rheology = rng.choice(["mevp", "mevp", "bbm"])
    precision = rng.choice(["fp64", "mixed"])
    mesh = rng.choice(["box", "quads", "sphere"] if rheology == "mevp" else ["box", "quads"])
    most = {"mevp": {"fp64": 250, "mixed": 500}, "bbm": {"fp64": 88, "mixed": 250}}[rheology][precision]
    if mesh != "box":
        most = min(most, 300)
    if mesh == "quads" and rheology == "bbm":
        most = min(most, 120)
    return _dyn(rheology, mesh, size(20, most), size(20, most), rng.choice([1, 3, 6]), precision)


# --- inputs --------------------------------------------------------------------


def _vertices(mesh, nx, ny):
    """Vertices ((nx+1)(ny+1), 2): the regular box, the box with displaced
    vertices (general quadrilaterals), or a lon/lat patch in radians."""
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1))
    if mesh == "sphere":
        step = 25e3 / 6371e3
        lon = (i - 0.5 * nx) * min(step, 0.6 / nx)
        lat = 1.0 + j * min(step, 0.3 / ny)
        return np.stack([lon.ravel(), lat.ravel()], axis=1)
    x, y = CELL * i, CELL * j
    if mesh == "quads":
        d = 0.04 * CELL * min(nx, ny)
        x = x + d * np.sin(3 * np.pi * i / nx) * np.sin(np.pi * j / ny)
        y = y + d * np.sin(2 * np.pi * j / ny) * np.sin(2 * np.pi * i / nx)
    return np.stack([x.ravel(), y.ravel()], axis=1)


def _mask(nx, ny):
    m = np.ones((ny, nx))
    m[0, :] = m[-1, :] = 0.0
    m[:, 0] = m[:, -1] = 0.0
    return m


def _fields(nx, ny, seed):
    """One model state and its forcing: thick and thin pack ice with ridges at
    cell scale, a cyclone, an ocean gyre, a wavy sea surface."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid((np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny)
    p = rng.uniform(0.0, 2.0 * np.pi, 6)
    wave = np.sin(4 * np.pi * x + p[0]) * np.cos(2 * np.pi * y + p[1])
    cx, cy = rng.uniform(0.35, 0.65, 2)
    dx, dy = (x - cx) * nx * CELL, (y - cy) * ny * CELL
    k = 4.0 / (nx * CELL)
    s = 15.0 * math.e * k * np.exp(-k * np.hypot(dx, dy))
    a = math.radians(72.0)
    f = {
        "hice": np.maximum(1.0 + 0.4 * wave + 0.02 * rng.standard_normal(x.shape), 0.0),
        "cice": np.clip(0.97 + 0.03 * np.cos(2 * np.pi * x + p[2]) + 0.005 * rng.standard_normal(x.shape), 0.0, 1.0),
        "damage": np.clip(1.0 - 0.05 * np.abs(rng.standard_normal(x.shape)), 0.0, 1.0),
        "u": 0.05 * np.sin(np.pi * x) * np.sin(2 * np.pi * y + p[3]),
        "v": 0.05 * np.sin(np.pi * y) * np.cos(2 * np.pi * x + p[4]),
        "uwind": -s * (math.cos(a) * dx + math.sin(a) * dy),
        "vwind": -s * (-math.sin(a) * dx + math.cos(a) * dy),
        "uocean": 0.1 * (2.0 * y - 1.0),
        "vocean": -0.1 * (2.0 * x - 1.0),
        "ssh": 0.05 * np.sin(2 * np.pi * x + p[5]) * np.sin(2 * np.pi * y),
    }
    return {n: np.ascontiguousarray(v.ravel()) for n, v in f.items()}


def _growth_fields(n, seed):
    rng = np.random.default_rng(seed)
    cice = rng.uniform(0.0, 1.0, n)
    cice[rng.random(n) < 0.05] = 0.0
    cice[rng.random(n) < 0.05] = 1.0
    hice = rng.uniform(0.0, 3.0, n) * cice
    hsnow = rng.uniform(0.0, 0.4, n) * cice
    hsnow[rng.random(n) < 0.2] = 0.0
    tf = rng.uniform(-1.9, -1.6, n)
    return {"hice": hice, "cice": cice, "hsnow": hsnow, "tice": rng.uniform(-30.0, 0.0, n),
            "qia": rng.uniform(-100.0, 400.0, n), "dqia_dt": rng.uniform(0.0, 30.0, n),
            "qow": rng.uniform(-200.0, 400.0, n), "qio": rng.uniform(0.0, 200.0, n),
            "sublim": rng.uniform(-1e-5, 1e-5, n),
            "snowfall": rng.uniform(0.0, 1e-4, n) * (rng.random(n) < 0.5), "penSW": rng.uniform(0.0, 50.0, n),
            "sst": tf + rng.uniform(-0.2, 2.0, n), "damage": rng.uniform(0.05, 1.0, n),
            "tf": tf, "mlbhc": 4186.84e3 * rng.uniform(5.0, 50.0, n)}


def _sides(case, seed):
    rng = np.random.default_rng(case["members"])  # the domains are the case's, the states the seed's
    return [tuple(int(v) for v in rng.integers(case["least"], case["most"] + 1, 2)) for _ in range(case["members"])]


# --- the package's calls ---------------------------------------------------------


def _kernel(rheology, mesh, nx, ny, dg, precision, f):
    cls = MEVPDynamicsKernel if rheology == "mevp" else BBMDynamicsKernel
    k = cls(dg_comp=dg, precision=int(precision == "mixed"), n_steps=SUB)
    k.initialise(_vertices(mesh, nx, ny), mesh == "sphere", _mask(nx, ny))
    for name in MODULE_IN + ("u", "v") + (("damage",) if rheology == "bbm" else ()):
        k.setData(name, f[name])
    return k


def prepare(case, seed):
    if case["kind"] == "growth":
        f = _growth_fields(case["cells"], seed)
        g = IceGrowth(case["cells"])
        for name in GROWTH_FIXED:
            g.setData(name, f[name])
        return {"kind": "growth", "growth": g, "in": f}
    if case["kind"] == "ensemble":
        members, ins = [], []
        for i, (nx, ny) in enumerate(_sides(case, seed)):
            f = _fields(nx, ny, seed * 101 + i)
            members.append(_kernel("mevp", "box", nx, ny, case["dg"], "mixed", f))
            ins.append({n: f[n] for n in ENSEMBLE_IN})
        outs = [{n: np.empty(m.nelements) for n in ENSEMBLE_OUT} for m in members]
        single = [{n: np.empty(m.nelements, dtype=np.float32) for n in ("u", "v")} for m in members]
        return {"kind": "ensemble", "ensemble": Ensemble(members), "members": members, "in": ins, "out": outs,
                "single": single, "t": 0.0}
    f = _fields(case["nx"], case["ny"], seed)
    k = _kernel(case["rheology"], case["mesh"], case["nx"], case["ny"], case["dg"], case["precision"], f)
    bbm = case["rheology"] == "bbm"
    n = case["nx"] * case["ny"]
    out = {name: np.empty(n) for name in MODULE_OUT + (("damage",) if bbm else ())}
    narrow = [name for name in out if name not in ("hice", "cice")] if case["precision"] == "mixed" else []
    return {"kind": "dynamics", "kernel": k, "in": {name: f[name] for name in MODULE_IN + (("damage",) if bbm else ())},
            "out": out, "single": {name: np.empty(n, dtype=np.float32) for name in narrow}, "t": 0.0}


def run(state):
    if state["kind"] == "growth":
        g, f = state["growth"], state["in"]
        for name in GROWTH_IN:
            g.setData(name, f[name])
        g.update(GROWTH_DT)
        return [g.getData(name) for name in GROWTH_OUT]
    if state["kind"] == "ensemble":
        for k, f in zip(state["members"], state["in"]):
            for name, a in f.items():
                k.setData(name, a)
        state["ensemble"].update(state["t"], DT)
        state["t"] += DT
        got = []
        for k, out, single in zip(state["members"], state["out"], state["single"]):
            for name, a in out.items():
                k.getDG0Data(name, a)
            for name, a in single.items():
                np.copyto(a, out[name], casting="same_kind")
            got.append([single.get(name, out[name]) for name in ENSEMBLE_OUT])
        return got
    out = state["kernel"].module_step(state["t"], DT, state["in"], state["out"])
    state["t"] += DT
    for name, a in state["single"].items():
        np.copyto(a, out[name], casting="same_kind")
    return [state["single"].get(name, a) for name, a in out.items()]


def work(case):
    """Bytes: the host fields in and out, and the device state of the step
    (fields, velocity, the element's stress terms, vertices), read and written
    once.  Flops: the products of the sub-cycle on the CG2 nodes' biquadratic
    velocity (a derivative and an interpolation per direction, forward and
    transposed), the rheology at nine Gauss points and the node update, and
    the advection."""
    if case["kind"] == "growth":
        return {"bytes": 8.0 * case["cells"] * (len(GROWTH_IN) + len(GROWTH_FIXED) + len(GROWTH_OUT)),
                "flops": 120.0 * case["cells"]}
    if case["kind"] == "ensemble":
        n = sum(nx * ny for nx, ny in _sides(case, 0))
        return {"bytes": n * (8.0 * (len(ENSEMBLE_IN) + len(ENSEMBLE_OUT)) + 8.0 * 4 * case["dg"] + 4.0 * (36 + 16)),
                "flops": n * (SUB * 900.0 + 4.0 * 60 * case["dg"])}
    n = case["nx"] * case["ny"]
    bbm = case["rheology"] == "bbm"
    real = 8.0 if case["precision"] == "fp64" else 4.0
    bytes_ = n * (8.0 * (len(MODULE_IN) + len(MODULE_OUT) + 2 * bbm) + 8.0 * (4 + 2 * bbm) * case["dg"] + 16.0
                  + real * ((48 if bbm else 36) + 16))
    return {"bytes": bytes_, "flops": n * (SUB * (1800.0 if bbm else 900.0) + 4.0 * 60 * case["dg"])}


# --- the same results in plain 64-bit torch / numpy ------------------------------

_P = dict(rho_ice=900.0, rho_atm=1.3, rho_ocean=1026.0, c_atm=1.2e-3, c_ocean=5.5e-3, fc=1.45842e-4, g=9.81,
          pstar=27500.0, delta_min=2e-9, alpha=1500.0, beta=1500.0)
_B = dict(compaction=-20.0, nu0=1.0 / 3.0, young=5.96e8, p0=10e3, lam=1e7, exp_relax=5.0, exp_compr=1.5,
          tan_phi=0.7, compr=1e10, c_lab=2e6)
_RADIUS = 6371000.0
_GAUSS = {1: ([0.5], [1.0]),
          2: ([0.5 - math.sqrt(1 / 12), 0.5 + math.sqrt(1 / 12)], [0.5, 0.5]),
          3: ([0.5 - math.sqrt(3 / 20), 0.5, 0.5 + math.sqrt(3 / 20)], [5 / 18, 8 / 18, 5 / 18]),
          4: ([0.5 + s * 0.5 * math.sqrt(3 / 7 + t * 2 / 7 * math.sqrt(6 / 5))
               for s, t in ((-1, 1), (-1, -1), (1, -1), (1, 1))],
              [(18 + t * math.sqrt(30)) / 72 for t in (-1, 1, 1, -1)])}


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _dg_basis(j, x, y, dx=0, dy=0):
    """The j-th DG basis function (or a first derivative) on the unit square."""
    x, y = x - 0.5, y - 0.5
    p, q = [(0, 0), (1, 0), (0, 1), (2, 0), (0, 2), (1, 1), (2, 1), (1, 2)][j]

    def one(n, t, d):
        return [[1.0 + 0 * t, t, t * t - 1 / 12], [0 * t, 1.0 + 0 * t, 2 * t]][d][n]
    return one(p, x, dx) * one(q, y, dy)


def _cg_basis(c, j, x, d=0):
    if c == 1:
        return [[1 - x, x], [-1 + 0 * x, 1 + 0 * x]][d][j]
    return [[2 * (x - 0.5) * (x - 1), 4 * x * (1 - x), 2 * x * (x - 0.5)], [4 * x - 3, 4 - 8 * x, 4 * x - 1]][d][j]


class _Mesh:
    """Geometry of the quadrilaterals at the Gauss points, in torch float64."""

    def __init__(self, mesh, nx, ny):
        self.nx, self.ny, self.n = nx, ny, nx * ny
        self.dev = _device()
        v = _vertices(mesh, nx, ny)
        self.sphere = mesh == "sphere"
        if self.sphere:  # the poles moved to Greenland and Antarctica
            lon, lat = v[:, 0], v[:, 1]
            x, y, z = np.cos(lat) * np.cos(lon), np.cos(lat) * np.sin(lon), np.sin(lat)
            a, b = math.radians(40.0), math.radians(15.0)
            x, y = math.cos(a) * x - math.sin(a) * y, math.sin(a) * x + math.cos(a) * y
            x, z = math.cos(b) * x - math.sin(b) * z, math.sin(b) * x + math.cos(b) * z
            v = np.stack([np.arctan2(y, x), np.arcsin(z)], axis=1)
        self.v = self.t(v).reshape(ny + 1, nx + 1, 2)
        self.ice = torch.tensor(_mask(nx, ny) == 1.0, device=self.dev)
        c = torch.stack([self.v[:-1, :-1], self.v[:-1, 1:], self.v[1:, :-1], self.v[1:, 1:]], 2).reshape(-1, 4, 2)
        if self.sphere:
            jump = (c[:, :1, 0] - c[:, :, 0]).abs().amax(1) > 2 / 3 * math.pi
            c[:, :, 0] += torch.where(jump[:, None] & (c[:, :, 0] < 0), 2 * math.pi, 0.0)
        self.corner = c
        ice = self.ice
        pad = torch.nn.functional.pad(ice, (1, 1, 1, 1))
        # closed sides: below, right, above, left
        self.closed = [ice & ~s for s in (pad[:-2, 1:-1], pad[1:-1, 2:], pad[2:, 1:-1], pad[1:-1, :-2])]
        self.zero = torch.zeros(2 * ny + 1, 2 * nx + 1, dtype=torch.bool, device=self.dev)
        for seg, places in enumerate((((0, 0), (0, 1), (0, 2)), ((0, 2), (1, 2), (2, 2)),
                                      ((2, 0), (2, 1), (2, 2)), ((0, 0), (1, 0), (2, 0)))):
            for r, k in places:
                self.zero[r:r + 2 * ny - 1:2, k:k + 2 * nx - 1:2] |= self.closed[seg]

    def t(self, a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)

    def points(self, q):
        p, w = _GAUSS[q]
        x, y = self.t(p * q), self.t([b for b in p for _ in range(q)])
        return x, y, self.t([a * b for b in w for a in w])

    def geometry(self, q):
        """Jacobian columns, determinant, weights and cos / sin of the latitude at q x q points."""
        x, y, w = self.points(q)
        fx = sum(self.corner[:, k, :, None] * (_cg_basis(1, k % 2, x, 1) * _cg_basis(1, k // 2, y)) for k in range(4))
        fy = sum(self.corner[:, k, :, None] * (_cg_basis(1, k % 2, x) * _cg_basis(1, k // 2, y, 1)) for k in range(4))
        lat = sum(self.corner[:, k, 1, None] * (_cg_basis(1, k % 2, x) * _cg_basis(1, k // 2, y)) for k in range(4))
        j = fx[:, 0] * fy[:, 1] - fx[:, 1] * fy[:, 0]
        one = torch.ones_like(j)
        return fx, fy, j, w, (lat.cos() if self.sphere else one), (lat.sin() if self.sphere else 0 * one)

    def psi(self, dg, q, dx=0, dy=0):
        x, y, _ = self.points(q)
        return torch.stack([_dg_basis(j, x, y, dx, dy) for j in range(dg)])

    def phi(self, c, q, dx=0, dy=0):
        x, y, _ = self.points(q)
        return torch.stack([_cg_basis(c, j % (c + 1), x, dx) * _cg_basis(c, j // (c + 1), y, dy)
                            for j in range((c + 1) ** 2)])

    def mass_inverse(self, dg):
        q = {1: 1, 3: 2}.get(dg, 3)
        _, _, j, w, cl, _ = self.geometry(q)
        p = self.psi(dg, q)
        return torch.linalg.inv(torch.einsum("iq,eq,jq->eij", p, j * w * cl, p))

    def gather(self, node):
        """The nine CG2 nodes of each element, (n, 9)."""
        return torch.stack([node[r:r + 2 * self.ny - 1:2, k:k + 2 * self.nx - 1:2]
                            for r in range(3) for k in range(3)], 2).reshape(self.n, 9)

    def scatter(self, el, c=2):
        """Sum of element contributions (n, (c+1)^2) at the CG nodes."""
        nx, ny = self.nx, self.ny
        out = torch.zeros(c * ny + 1, c * nx + 1, dtype=torch.float64, device=self.dev)
        el = el.reshape(ny, nx, -1)
        for r in range(c + 1):
            for k in range(c + 1):
                out[r:r + c * ny - c + 1:c, k:k + c * nx - c + 1:c] += el[:, :, r * (c + 1) + k]
        return out

    def to_nodes(self, f, c=2):
        """A DG field (n, dg) averaged to the CG nodes."""
        p = torch.linspace(0, 1, c + 1, dtype=torch.float64, device=self.dev)
        x, y = p.repeat(c + 1), p.repeat_interleave(c + 1)
        at = f @ torch.stack([_dg_basis(j, x, y) for j in range(f.shape[1])])
        share = torch.ones(c + 1, dtype=torch.float64, device=self.dev)
        share[0] = share[-1] = 0.5
        out = self.scatter(at * (share[:, None] * share[None, :]).reshape(-1), c)
        for edge in (out[0], out[-1], out[:, 0], out[:, -1]):
            edge *= 2.0
        return out

    def to_dg(self, node, dg, minv):
        q = {1: 1, 3: 2}.get(dg, 3)
        _, _, j, w, cl, _ = self.geometry(q)
        val = self.gather(node) @ self.phi(2, q)
        return torch.einsum("eij,ej->ei", minv, (val * j * w * cl) @ self.psi(dg, q).T)


def _traces(f, side):
    """A cell's polynomial on a side (below, right, above, left)."""
    n = f.shape[-1]
    z = f.new_zeros(f.shape[:-1])
    c = [f[..., j] if j < n else z for j in range(8)]
    s = 0.5 if side in (1, 2) else -0.5
    if side in (1, 3):
        t = [c[0] + s * c[1] + c[3] / 6, c[2] + s * c[5] + c[6] / 6, c[4] + s * c[7]]
    else:
        t = [c[0] + s * c[2] + c[4] / 6, c[1] + s * c[5] + c[7] / 6, c[3] + s * c[6]]
    return torch.stack(t[:{1: 1, 3: 2}.get(n, 3)], -1)


class _Advection:
    """Upwind DG transport with the second-order Runge-Kutta scheme."""

    def __init__(self, m, dg, ux, uy):
        self.m, self.dg = m, dg
        self.q = {1: 1, 3: 2}.get(dg, 3)
        fx, fy, _, w, _, _ = m.geometry(self.q)
        px, py = m.psi(dg, self.q, 1, 0), m.psi(dg, self.q, 0, 1)
        self.cx = (px * fy[:, None, 1] - py * fx[:, None, 1]) * w
        self.cy = (py * fx[:, None, 0] - px * fy[:, None, 0]) * w
        minv = m.mass_inverse(dg)
        self.minv = minv / _RADIUS if m.sphere else minv
        self.vel = (m.to_dg(ux, dg, minv), m.to_dg(uy, dg, minv))
        g = m.t(_GAUSS[self.q][0])
        self.edge = torch.stack([_dg_basis(j, g, 0 * g + 0.5) for j in (0, 1, 3)[:self.q]])  # 1-D basis at the points
        gw = m.t(_GAUSS[self.q][1])
        self.back = [torch.stack([gw * _dg_basis(j, *p) for j in range(dg)])
                     for p in ((g, 0 * g), (0 * g + 1, g), (g, 0 * g + 1), (0 * g, g))]
        vx, vy = (a.reshape(m.ny, m.nx, dg) * m.ice[..., None] for a in self.vel)
        along = m.v[:, 1:] - m.v[:, :-1], m.v[1:] - m.v[:-1]
        if m.sphere:
            along = tuple(torch.stack([torch.remainder(a[..., 0] + math.pi, 2 * math.pi) - math.pi, a[..., 1]], -1)
                          for a in along)
        tx, ty = along
        nX = torch.zeros(m.ny + 1, m.nx, self.q, dtype=torch.float64, device=m.dev)
        nY = torch.zeros(m.ny, m.nx + 1, self.q, dtype=torch.float64, device=m.dev)
        for s, side in ((slice(0, -1), 0), (slice(1, None), 2)):
            t = tx[s]
            nX[s] += 0.5 * (t[..., :1] * _traces(vy, side) - t[..., 1:] * _traces(vx, side))
        for s, side in ((slice(0, -1), 3), (slice(1, None), 1)):
            t = ty[:, s]
            nY[:, s] += 0.5 * (t[..., 1:] * _traces(vx, side) - t[..., :1] * _traces(vy, side))
        for seg, where in ((0, nX[:-1]), (2, nX[1:]), (1, nY[:, 1:]), (3, nY[:, :-1])):
            where *= torch.where(m.closed[seg], 2.0, 1.0)[..., None]
        self.gX, self.gY = nX @ self.edge, nY @ self.edge
        p = m.psi(dg, self.q)
        self.p, self.vg = p, (self.vel[0] @ p, self.vel[1] @ p)

    def rhs(self, dt, f):
        m = self.m
        pg = f @ self.p
        up = dt * torch.einsum("eiq,eq->ei", self.cx * self.vg[0][:, None] + self.cy * self.vg[1][:, None], pg)
        if self.dg == 1:
            up = 0 * up
        up = up.reshape(m.ny, m.nx, -1) * m.ice[..., None]
        f = f.reshape(m.ny, m.nx, -1)
        tr = [_traces(f, s) @ self.edge for s in range(4)]

        def upwind(v, low, high, both):
            return (v.clamp(min=0) * low + v.clamp(max=0) * high) * both[..., None]
        flux = upwind(self.gY[:, 1:-1], tr[1][:, :-1], tr[3][:, 1:], m.ice[:, :-1] & m.ice[:, 1:])
        up[:, :-1] -= dt * flux @ self.back[1].T
        up[:, 1:] += dt * flux @ self.back[3].T
        flux = upwind(self.gX[1:-1], tr[2][:-1], tr[0][1:], m.ice[:-1] & m.ice[1:])
        up[:-1] -= dt * flux @ self.back[2].T
        up[1:] += dt * flux @ self.back[0].T
        for seg, v in ((0, -self.gX[:-1]), (1, self.gY[:, 1:]), (2, self.gX[1:]), (3, -self.gY[:, :-1])):
            up -= dt * (tr[seg] * v.clamp(min=0) * m.closed[seg][..., None]) @ self.back[seg].T
        return torch.einsum("eij,ej->ei", self.minv, up.reshape(m.n, -1))

    def step(self, dt, f):
        k = self.rhs(dt, f)
        return f + k + 0.5 * (self.rhs(dt, f + k) - k)


def _limit(m, f, lo=None, hi=None):
    f = f.clone()
    for bound, sign in ((hi, 1.0), (lo, -1.0)):
        if bound is None:
            continue
        f[:, 0] = f[:, 0].clamp(max=bound) if sign > 0 else f[:, 0].clamp(min=bound)
        room = sign * (bound - f[:, 0])
        if f.shape[1] == 3:
            over = 2.0 * torch.maximum((f[:, 1] + f[:, 2]).abs(), (f[:, 1] - f[:, 2]).abs())
        elif f.shape[1] == 6:
            over = ((sign * (f @ m.psi(6, 3))).amax(1)) - sign * f[:, 0]
        else:
            continue
        scale = torch.where(over > room, room / torch.where(over == 0, torch.ones_like(over), over),
                            torch.ones_like(over))
        f[:, 1:] *= scale[:, None]
    return f


def _ssh_gradient(m, ssh):
    fx, fy, _, w, cl, _ = m.geometry(3)
    px, py, p = m.phi(1, 3, 1, 0), m.phi(1, 3, 0, 1), m.phi(1, 3)
    gx = (px * fy[:, None, 1] - py * fx[:, None, 1]) * w
    gy = (py * fx[:, None, 0] - px * fy[:, None, 0]) * w * cl[:, None]
    node = m.to_nodes(ssh[:, None], 1)
    loc = torch.stack([node[:-1, :-1], node[:-1, 1:], node[1:, :-1], node[1:, 1:]], 2).reshape(m.n, 4) @ p
    r = _RADIUS if m.sphere else 1.0
    _, _, j, w2, cl2, _ = m.geometry(2)
    lumped = m.scatter((j * w2 * cl2) @ m.phi(1, 2).T, 1)
    out = []
    for g in (gx, gy):
        d = -m.scatter(torch.einsum("eiq,eq->ei", g, loc) / r, 1) / lumped
        d[0], d[-1] = d[1].clone(), d[-2].clone()
        d[:, 0], d[:, -1] = d[:, 1].clone(), d[:, -2].clone()
        full = torch.zeros(2 * m.ny + 1, 2 * m.nx + 1, dtype=torch.float64, device=m.dev)
        full[::2, ::2] = d
        full[::2, 1::2] = 0.5 * (d[:, :-1] + d[:, 1:])
        full[1::2, ::2] = 0.5 * (d[:-1] + d[1:])
        full[1::2, 1::2] = 0.25 * (d[:-1, :-1] + d[:-1, 1:] + d[1:, :-1] + d[1:, 1:])
        out.append(full)
    return out


def _exact_dynamics(case, f):
    m = _Mesh(case["mesh"], case["nx"], case["ny"])
    dg, n, bbm = case["dg"], m.n, case["rheology"] == "bbm"
    fo, fa = _P["c_ocean"] * _P["rho_ocean"], _P["c_atm"] * _P["rho_atm"]

    def dg0(name):
        a = torch.zeros(n, dg, dtype=torch.float64, device=m.dev)
        a[:, 0] = m.t(f[name])
        return a
    u, v, ua, va, uo, vo = (m.to_nodes(dg0(k)) for k in ("u", "v", "uwind", "vwind", "uocean", "vocean"))
    # the brittle kernel advects with its sub-cycle averages, zero before the first step
    adv = _Advection(m, dg, *((0 * u, 0 * v) if bbm else (u, v)))
    A = _limit(m, adv.step(DT, dg0("cice")), 0.0, 1.0)
    H = _limit(m, adv.step(DT, dg0("hice")), 0.0)
    D = _limit(m, adv.step(DT, dg0("damage")), 1e-12, 1.0) if bbm else None
    cA, cH = m.to_nodes(A).clamp(1e-4, 1.0), m.to_nodes(H).clamp(min=1e-4)
    gu, gv = _ssh_gradient(m, m.t(f["ssh"]))

    fx, fy, j, w, cl, sl = m.geometry(3)
    r = _RADIUS if m.sphere else 1.0
    px, py, p8 = m.phi(2, 3, 1, 0), m.phi(2, 3, 0, 1), m.psi(8, 3)
    gx = (px * fy[:, None, 1] - py * fx[:, None, 1]) * w
    gy = (py * fx[:, None, 0] - px * fy[:, None, 0]) * w * cl[:, None]
    d1, d2 = torch.einsum("ejq,kq->ejk", gx, p8) / r, torch.einsum("ejq,kq->ejk", gy, p8) / r
    dm = torch.einsum("jq,eq,kq->ejk", m.phi(2, 3), j * sl * w, p8) / r
    minv8 = m.mass_inverse(8)
    strain = [torch.einsum("kq,ekl,ejl->eqj", p8, minv8, d) for d in (d1, d2, dm)]
    project = torch.einsum("ekl,lq,eq->ekq", minv8, p8, j * w)
    _, _, j4, w4, cl4, _ = m.geometry(4)
    lumped = m.scatter((j4 * w4 * cl4) @ m.phi(2, 4).T)
    p3 = m.psi(dg, 3)
    hq, aq = (H @ p3).clamp(min=0), (A @ p3).clamp(0, 1)
    land = (~m.ice).reshape(-1)
    for s in strain:
        s[land] = 0.0
    s11, s12, s22 = (torch.zeros(n, 8, dtype=torch.float64, device=m.dev) for _ in range(3))

    def mv(op, a):
        return torch.einsum("eqj,ej->eq", op, a)

    def strains():
        ul, vl = m.gather(u), m.gather(v)
        e11, e22, e12 = mv(strain[0], ul), mv(strain[1], vl), 0.5 * (mv(strain[0], vl) + mv(strain[1], ul))
        if m.sphere:
            e11, e12 = e11 - mv(strain[2], vl), e12 + 0.5 * mv(strain[2], ul)
        return e11, e12, e22

    def divergence():
        tx, ty = mv(d1, s11) + mv(d2, s12), mv(d1, s12) + mv(d2, s22)
        if m.sphere:
            tx, ty = tx + mv(dm, s12), ty - mv(dm, s11)
        out = []
        for t in (tx, ty):
            t = torch.where(land[:, None], 0.0, t)
            out.append(torch.where(m.zero, 0.0, -m.scatter(t)) / lumped)
        return out

    rho_h = _P["rho_ice"] * cH
    wind = torch.sqrt(ua * ua + va * va)
    mean_u, mean_v = torch.zeros_like(u), torch.zeros_like(v)
    u0, v0 = u, v
    if bbm:
        dt = DT / SUB
        damage = D
        size = torch.sqrt(_area(m))
        dam_minv = m.mass_inverse(dg)
        dam_project = torch.einsum("ekl,lq,eq->ekq", dam_minv, p3, j * w)
        ex = torch.exp(_B["compaction"] * (1 - aq))
        pmax = _B["p0"] * hq ** (_B["exp_compr"] + 1) * ex
        scale = torch.sqrt(0.1 / size)[:, None]
    else:
        P = _P["pstar"] * hq * torch.exp(-20.0 * (1.0 - aq))
    for _ in range(SUB):
        e11, e12, e22 = strains()
        if bbm:
            g11, g12, g22 = s11 @ p8, s12 @ p8, s22 @ p8
            d = (damage @ p3).clamp(1e-12, 1.0)
            sn = 0.5 * (g11 + g22)
            tv = _B["lam"] * (d * ex) ** (_B["exp_relax"] - 1)
            tp = torch.where(sn < 0, (-pmax / torch.where(sn < 0, sn, -1.0)).clamp(max=1.0), 0.0)
            mult = tv / (tv + (1 - tp) * dt)
            el = hq * _B["young"] * d * ex
            k = dt * el / (1 - _B["nu0"] ** 2)
            g11 = (g11 + k * (e11 + _B["nu0"] * e22)) * mult
            g22 = (g22 + k * (_B["nu0"] * e11 + e22)) * mult
            g12 = (g12 + k * e12 * (1 - _B["nu0"])) * mult
            sn = 0.5 * (g11 + g22)
            tau = torch.sqrt(0.25 * (g11 - g22) ** 2 + g12 * g12)
            mc = tau + _B["tan_phi"] * sn
            crit = torch.where(mc > 0, _B["c_lab"] * scale * hq / torch.where(mc > 0, mc, 1.0), 1.0)
            cs = _B["compr"] * scale * hq
            crit = torch.where(sn < -cs, -cs / torch.where(sn < -cs, sn, -1.0), crit).clamp(max=1.0)
            td = size[:, None] * math.sqrt(2 * (1 + _B["nu0"]) * _P["rho_ice"]) / torch.sqrt(el)
            keep = 1 - (1 - crit) * dt / td
            damage = mv(dam_project, d * keep)
            s11, s12, s22 = mv(project, g11 * keep), mv(project, g12 * keep), mv(project, g22 * keep)
        else:
            delta = torch.sqrt(_P["delta_min"] ** 2 + 1.25 * (e11 ** 2 + e22 ** 2) + 1.5 * e11 * e22 + e12 ** 2)
            z, a = P / 8 / delta, 1 / _P["alpha"]
            s11 = (1 - a) * s11 + a * mv(project, z * (5 * e11 + 3 * e22) - 0.5 * P)
            s22 = (1 - a) * s22 + a * mv(project, z * (5 * e22 + 3 * e11) - 0.5 * P)
            s12 = (1 - a) * s12 + a * mv(project, 2 * z * e12)
        dx, dy = divergence()
        slip = torch.sqrt((uo - u) ** 2 + (vo - v) ** 2)
        if bbm:
            c = dt / rho_h
            cp = cA * fo * slip
            al, be = 1 + c * cp, dt * _P["fc"]
            den = 1 / (al * al + be * be)
            fxn = dx - rho_h * _P["g"] * gu + cA * fa * wind * ua + cp * uo
            fyn = dy - rho_h * _P["g"] * gv + cA * fa * wind * va + cp * vo
            u, v = ((al * u + be * v + c * (al * fxn + be * fyn)) * den,
                    (al * v - be * u + c * (al * fyn + be * fxn)) * den)
            mean_u, mean_v = mean_u + u / SUB, mean_v + v / SUB
        else:
            c = rho_h / DT
            den = 1 / (c * (1 + _P["beta"]) + cA * fo * slip)
            u, v = (den * (c * (_P["beta"] * u + u0) + cA * (fa * wind * ua + fo * slip * uo) - rho_h * _P["fc"] * u
                           - rho_h * _P["g"] * gu + dx),
                    den * (c * (_P["beta"] * v + v0) + cA * (fa * wind * va + fo * slip * vo) + rho_h * _P["fc"] * v
                           - rho_h * _P["g"] * gv + dy))
        u, v = torch.where(m.zero, 0.0, u), torch.where(m.zero, 0.0, v)
    if bbm:
        rel = uo - mean_u, vo - mean_v
    else:
        rel = u - uo, v - vo
    drag = fo * torch.sqrt(rel[0] ** 2 + rel[1] ** 2)
    minv = m.mass_inverse(dg)
    nodes = [m.to_dg(a, dg, minv)[:, 0] for a in (u, v, drag * rel[0], drag * rel[1])]
    out = {"hice": H[:, 0], "cice": A[:, 0], "u": nodes[0], "v": nodes[1], "uiostress": nodes[2],
           "viostress": nodes[3]}
    if bbm:
        out["damage"] = damage[:, 0]
    return {k: a.cpu().numpy() for k, a in out.items()}


def _area(m):
    c = m.corner

    def sq(a, b):
        return ((c[:, a] - c[:, b]) ** 2).sum(1)
    t = sq(1, 3) + sq(0, 2) - sq(0, 1) - sq(2, 3)
    return 0.25 * torch.sqrt(4 * sq(0, 3) * sq(1, 2) - t * t)


def _exact_growth(f):
    """IceGrowth with its default modules (ThermoIce0, HiblerSpread,
    ConstantHealing) in numpy."""
    lf, rho_i, rho_s, rho_o, kappa, ks, h_min, c_min = 333.55e3, 917.0, 330.0, 1025.0, 2.0334, 0.3096, 0.01, 1e-12
    dt, qow, qio = GROWTH_DT, f["qow"].copy(), f["qio"].copy()
    with np.errstate(all="ignore"):
        some = (f["cice"] > 0) & (f["hice"] > 0)
        cice = np.where(some, f["cice"], 0.0)
        hice = np.where(some, f["hice"] / f["cice"], 0.0)
        hsnow = np.where(some, f["hsnow"] / f["cice"], 0.0)
        h0, tice0 = hice.copy(), f["tice"]

        def minimum(hice, cice, hsnow, qow):
            small = ((0 < cice) & (cice < c_min)) | ((0 < hice) & (hice < h_min))
            qow = np.where(small, qow + cice * lf * (hice * rho_i + hsnow * rho_s) / dt, qow)
            return np.where(small, 0, hice), np.where(small, 0, cice), np.where(small, 0, hsnow), qow
        hice, cice, hsnow, qow = minimum(hice, cice, hsnow, qow)
        on = (hice != 0) & (cice != 0)
        slab = ks * kappa / (ks * hice + kappa * hsnow) * 1.065
        qic = slab * (f["tf"] - tice0)
        left = qic - (f["qia"] + 0.6 * f["penSW"])
        tice = np.minimum(np.where(hsnow > 0, 0.0, -0.055 * 5), tice0 + left / (slab + f["dqia_dt"]))
        melt = np.minimum(-left, 0.0) / (lf * rho_s)
        snow = hsnow + (melt - f["sublim"] / rho_s) * dt
        excess = np.minimum(snow, 0.0) * rho_s / rho_i
        snow = np.maximum(snow, 0.0)
        dh = excess + (qic - qio) * dt / (lf * rho_i)
        h = hice + dh
        snow = np.where(h > 0, snow + f["snowfall"] * dt / rho_s, snow)
        draught = (h * rho_i + snow * rho_s) / rho_o
        flood = draught > h
        snow = np.where(flood, snow - (draught - h) * rho_i / rho_s, snow)
        h = np.where(flood, draught, h)
        gone = on & (h < h_min)
        qio = np.where(gone, qio + h * lf * rho_i / dt + snow * lf * rho_s / dt, qio)
        dh = np.where(gone, -h0, dh)
        dh = np.where(on, dh, 0.0)
        tice = np.where(on, np.where(gone, 0.0, tice), tice0)
        hice = np.where(on, np.where(gone, 0.0, h), hice)
        hsnow = np.where(on, np.where(gone, 0.0, snow), hsnow)
        cice = np.where(gone, 0.0, cice)
        cool = -qow / f["mlbhc"] * dt
        new = f["sst"] + cool < f["tf"]
        sensible = (f["tf"] - f["sst"]) / cool * qow
        newice = np.where(new, (qow - sensible) * dt * (1 - cice) / (lf * rho_i), 0.0)
        qow = np.where(new, sensible, qow)
        dc = newice * (1.0 / 0.25) + np.where((dh < 0) & (cice < 1), dh * cice * 0.5 / h0, 0.0)
        cice = np.where((hice > 0) | (newice > 0), cice + dc, 0.0)
        wide = cice >= c_min
        hice = np.where(wide, hice + (newice - hice * dc) / cice, hice)
        qow = np.where(wide & (dc < 0), qow - dc * hsnow * lf * rho_s / dt, qow)
        hsnow = np.where(wide & ~(dc < 0), hsnow - hsnow * dc / cice, hsnow)
        hice, cice, hsnow, qow = minimum(hice, cice, hsnow, qow)
        grown = np.maximum(0.0, dc)
        healed = (f["damage"] * (cice - grown) + grown) / cice + dt / (15.0 * 86400.0)
        damage = np.where(healed < 1.0, healed, 1.0)
    got = {"hice_updated": hice, "cice_updated": cice, "hsnow_updated": hsnow, "tice_updated": tice,
           "newice": newice, "qow": qow, "qio": qio, "damage": damage}
    return [got[name] for name in GROWTH_OUT]


def exact(case, seed):
    if case["kind"] == "growth":
        return _exact_growth(_growth_fields(case["cells"], seed))
    if case["kind"] == "ensemble":
        got = []
        for i, (nx, ny) in enumerate(_sides(case, seed)):
            e = _exact_dynamics(_dyn("mevp", "box", nx, ny, case["dg"], "mixed"), _fields(nx, ny, seed * 101 + i))
            got.append([e[name] for name in ENSEMBLE_OUT])
        return got
    e = _exact_dynamics(case, _fields(case["nx"], case["ny"], seed))
    return [e[name] for name in MODULE_OUT + (("damage",) if case["rheology"] == "bbm" else ())]
