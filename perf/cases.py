"""The work that users of this framework have it do, as cases that can be timed.

A case is a plain dict; ``prepare`` builds what a driver script holds before its
loop (model, state, host buffers), ``run`` is one pass through the public API
(``advance``, ``residual_norms``, ``step``, ``get_field``) as a driver calls it, and
``exact`` is the same pass in 64-bit torch, written here from the discrete
equations.  Fields of FullStokes models are read in place through
``device_ptr`` / ``layout``; immersed-boundary and heat models are read back with
``get_field`` (a state pointer handed out would switch off the immersed-boundary
model's skipping of inactive points).

Families:

* ``slab``       3D gravity-driven slab: Glen n = 3, periodic x / y, slip bed, free top
* ``mms3d``      3D manufactured-solution box: linear viscosity, slip walls, body-force fields
* ``plane``      2D models: the unit-square manufactured solution, or a Glen flow on a frozen bed
* ``glacier``    3D immersed-boundary ice between a bumpy bed and a surface
* ``inclusions`` a batch of 2D pure-shear models with circular inclusions
* ``glaciers``   a batch of small 3D immersed-boundary glaciers
* ``heat``       an implicit step of 3D heat diffusion
"""
import gc
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DTYPES = {"f64": (torch.float64, np.float64, 8), "f32": (torch.float32, np.float32, 4)}
F3 = ("P", "txx", "tyy", "tzz", "txy", "txz", "tyz", "Vx", "Vy", "Vz")
F2 = ("P", "txx", "tyy", "txy", "Vx", "Vy")
# staggered location of each field, (x, y, z): 0 cell centre, 1 vertex
LOC = {"P": (0, 0, 0), "txx": (0, 0, 0), "tyy": (0, 0, 0), "tzz": (0, 0, 0), "txy": (1, 1, 0), "txz": (1, 0, 1),
       "tyz": (0, 1, 1), "Vx": (1, 0, 0), "Vy": (0, 1, 0), "Vz": (0, 0, 1), "eta": (0, 0, 0)}


def _package():
    """The framework's Python package (its folder's name is not an identifier)."""
    name = "fastice_b200"
    if name not in sys.modules:
        pkg = os.path.join(ROOT, "fastice.jl_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# ---- the cases ---------------------------------------------------------------------
def listed():
    return [
        # the slab at the size the benchmark quotes, both precisions: production sweeps
        {"name": "slab511_f64", "family": "slab", "nx": 511, "ny": 511, "nz": 511, "dtype": "f64", "iters": 6,
         "rounds": 1, "norms": False},
        {"name": "slab511_f32", "family": "slab", "nx": 511, "ny": 511, "nz": 511, "dtype": "f32", "iters": 6,
         "rounds": 1, "norms": False},
        # an ordinary slab whose sides are no multiples of any tile, with the driver's check
        {"name": "slab_ragged_f64", "family": "slab", "nx": 259, "ny": 193, "nz": 125, "dtype": "f64", "iters": 24,
         "rounds": 1, "norms": True},
        # the smallest 3D runs (set-ups, regression runs): launches and latency count
        {"name": "slab_small_f64", "family": "slab", "nx": 47, "ny": 33, "nz": 29, "dtype": "f64", "iters": 64,
         "rounds": 1, "norms": True},
        # the 3D convergence study: walls on every side, two checks of the driver loop
        {"name": "mms3d_127_f64", "family": "mms3d", "nx": 127, "ny": 127, "nz": 127, "dtype": "f64", "iters": 127,
         "rounds": 2, "norms": True},
        # the 2D convergence study at the size its tests use
        {"name": "mms2d_128_f64", "family": "plane", "kind": "mms", "nx": 128, "ny": 128, "dtype": "f64",
         "iters": 128, "rounds": 4, "norms": True},
        # a large 2D section with Glen's law
        {"name": "glen2d_1021x509_f64", "family": "plane", "kind": "glen", "nx": 1021, "ny": 509, "dtype": "f64",
         "iters": 256, "rounds": 1, "norms": True},
        # the glacier at full size, one check-to-check round
        {"name": "glacier383_f64", "family": "glacier", "nx": 383, "ny": 383, "nz": 383, "dtype": "f64",
         "iters": 383, "rounds": 1},
        # the single-precision sweeps of a mixed-precision glacier solve
        {"name": "glacier191_f32", "family": "glacier", "nx": 191, "ny": 191, "nz": 191, "dtype": "f32",
         "iters": 191, "rounds": 2},
        # an ensemble of uneven 2D instances between two checks
        {"name": "inclusions48_f32", "family": "inclusions", "members": 48, "lo": 63, "hi": 511, "draw": 7,
         "dtype": "f32", "iters": 256},
        # an ensemble of small glaciers
        {"name": "glaciers12_f64", "family": "glaciers", "members": 12, "lo": 16, "hi": 48, "draw": 3,
         "dtype": "f64", "iters": 256},
        # one implicit step of heat diffusion
        {"name": "heat255_f64", "family": "heat", "nx": 255, "ny": 255, "nz": 255, "dtype": "f64", "iters": 400},
    ]


def _odd_dims(rng, lo, hi, nd, spread=1.7, least=12):
    """Sides of about c**(1/nd) cells each, c log-uniform, uneven and of either parity."""
    side = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return [max(least, min(int(round(hi * 1.3)), int(round(side * math.exp(rng.uniform(-1, 1) * math.log(spread) / 2)))))
            for _ in range(nd)]


def draw(rng):
    family = rng.choice(["slab", "slab", "mms3d", "plane", "plane", "glacier", "inclusions", "glaciers", "heat"])
    dtype = rng.choice(["f64", "f64", "f32"])
    if family in ("slab", "mms3d"):
        d = _odd_dims(rng, 24, 400 if family == "slab" else 200, 3)
        most = 6e8 / (d[0] * d[1] * d[2])
        return {"family": family, "nx": d[0], "ny": d[1], "nz": d[2], "dtype": dtype,
                "iters": max(4, min(rng.randint(8, 128), int(most))), "rounds": 1, "norms": True}
    if family == "plane":
        d = _odd_dims(rng, 48, 1100, 2, spread=2.0)
        return {"family": "plane", "kind": rng.choice(["mms", "glen"]), "nx": d[0], "ny": d[1], "dtype": dtype,
                "iters": rng.randint(48, 256), "rounds": rng.randint(1, 3), "norms": True}
    if family == "glacier":
        d = _odd_dims(rng, 40, 255, 3, spread=1.3)
        return {"family": "glacier", "nx": d[0], "ny": d[1], "nz": d[2], "dtype": dtype,
                "iters": rng.randint(64, 200), "rounds": 1}
    if family == "inclusions":
        return {"family": "inclusions", "members": rng.randint(8, 48), "lo": rng.choice([31, 63]),
                "hi": rng.choice([255, 511]), "draw": rng.randint(0, 10 ** 6), "dtype": dtype,
                "iters": 2 * rng.randint(32, 128)}
    if family == "glaciers":
        return {"family": "glaciers", "members": rng.randint(3, 16), "lo": rng.randint(12, 24),
                "hi": rng.randint(32, 64), "draw": rng.randint(0, 10 ** 6), "dtype": dtype,
                "iters": rng.randint(64, 256)}
    d = _odd_dims(rng, 40, 255, 3)
    return {"family": "heat", "nx": d[0], "ny": d[1], "nz": d[2], "dtype": dtype, "iters": rng.randint(64, 400)}


def _members(case):
    """Grid sides of a batch's members: uneven, fixed by the case."""
    rng = random.Random(case["draw"])
    nd = 2 if case["family"] == "inclusions" else 1
    return [tuple(rng.randint(case["lo"], case["hi"]) for _ in range(nd)) for _ in range(case["members"])]


def work(case):
    esz = DTYPES[case["dtype"]][2]
    fam, its = case["family"], case["iters"] * case.get("rounds", 1)
    if fam in ("slab", "mms3d"):
        n = (case["nx"], case["ny"], case["nz"])
        # P, six stresses and three velocities read and written, viscosity read and written
        e = sum(2 * _count(n, LOC[f]) for f in F3 + ("eta",))
        e += sum(_count(n, LOC[f]) for f in ("Vx", "Vy", "Vz")) if fam == "mms3d" else 0  # body force
        return {"bytes": float(e * esz * its), "flops": 150.0 * n[0] * n[1] * n[2] * its}
    if fam == "plane":
        n = (case["nx"], case["ny"], 1)
        e = 14 if case["kind"] == "glen" else 15
        return {"bytes": float(e * n[0] * n[1] * esz * its), "flops": 70.0 * n[0] * n[1] * its}
    if fam == "inclusions":
        c = sum(a * b for a, b in _members(case))
        return {"bytes": 13.0 * c * esz * its, "flops": 60.0 * c * its}
    if fam == "heat":
        c = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": (9.0 * its + 1) * c * esz, "flops": 40.0 * c * its}
    # about a quarter of the box is ice: ten state fields read and written, the viscosity
    # and seven volume fractions read there, and an activity byte per point
    c = sum(a ** 3 for a, in _members(case)) if fam == "glaciers" else case["nx"] * case["ny"] * case["nz"]
    return {"bytes": (28 * 0.25 * esz + 1.0) * c * its, "flops": 200.0 * 0.25 * c * its}


def _count(n, loc):
    return math.prod(a + b for a, b in zip(n, loc))


# ---- inputs ------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pt_steps(extent, dims, r=0.7, re=8 * math.pi, factor=1.1):
    """Pseudo-transient steps as the drivers compute them."""
    nd = len(dims)
    ltau = min(extent) / re
    vdtau = min(e / n for e, n in zip(extent, dims)) / math.sqrt(nd * factor)
    theta = ltau * (r + 4 / 3) / vdtau
    taus = ("xx", "yy", "zz", "xy", "xz", "yz") if nd == 3 else ("xx", "yy", "xy")
    return {"Δτ": {"Pr": r / theta, "τ": {k: 1.0 / (theta + 1.0) for k in taus},
                   "V": {k: vdtau * ltau for k in ("x", "y", "z")[:nd]}}}


def _coord(n, extent, loc, origin=0.0):
    """Interior coordinates along one dimension."""
    h = extent / n
    return origin + h * (torch.arange(n + loc, dtype=torch.float64, device=_device()) + (0.0 if loc else 0.5))


def _smooth(rs, dims, extent, loc, amplitude, modes=3):
    """A smooth field, periodic in x and y: a few products of waves with seeded phases."""
    out = None
    for _ in range(modes):
        f = None
        for d in range(len(dims)):
            k = 2 * math.pi / extent[d] * int(rs.randint(1, 4)) * (1.0 if d < 2 else 0.5)
            w = torch.sin(k * _coord(dims[d], extent[d], loc[d]) + float(rs.uniform(0, 2 * math.pi)))
            f = w if f is None else w.reshape((-1,) + (1,) * d) * f
        f = f * (amplitude * float(rs.uniform(0.5, 1.0)) / modes)
        out = f if out is None else out.add_(f)
    return out


def _rounded(t, dtype):
    return t.to(DTYPES[dtype][0]).to(torch.float64)


def _start3(case, seed, extent, v, tau, p):
    """A state in the middle of a solve, generated field by field as (name, values)."""
    n = (case["nx"], case["ny"], case["nz"])
    rs = np.random.RandomState(seed % (1 << 31))
    for f in F3:
        yield f, _rounded(_smooth(rs, n, extent, LOC[f], v if f[0] == "V" else p if f == "P" else tau), case["dtype"])


def _slab(case, seed):
    extent = (1.0, 1.0, 0.25)
    n = (case["nx"], case["ny"], case["nz"])
    a = math.radians(10.0)
    rs = np.random.RandomState((seed + 77) % (1 << 31))
    return {"nd": 3, "n": n, "extent": extent, "steps": _pt_steps(extent, n), "gravity": (-math.sin(a), 0.0, math.cos(a)),
            "bcs": (("periodic", "periodic"), ("periodic", "periodic"), ("slip", "traction")), "glen": (1.0, 5000.0),
            "eta": _rounded(4000.0 * torch.exp(_smooth(rs, n, extent, LOC["eta"], 0.4)), case["dtype"])}


def _mms_f(a, b):
    return np.cos(math.pi * a) * (b ** 2 - 1) ** 2 - np.cos(math.pi * b) * (a ** 2 - 1) ** 2


def _mms_p(a, b):
    return np.cos(math.pi * b) * (1 - 3 * a ** 2) * 2 - np.cos(math.pi * a) * (1 - 3 * b ** 2) * 2


def _mms3d(case, seed):
    """Free-slip walls and the body force of a divergence-free manufactured velocity."""
    n, extent = (case["nx"], case["ny"], case["nz"]), (2.0, 2.0, 2.0)
    scale = float(np.random.RandomState((seed + 77) % (1 << 31)).uniform(0.5, 2.0))
    g = []
    for c in range(3):
        loc = [1 if d == c else 0 for d in range(3)]
        z, y, x = np.meshgrid(*[_coord(n[d], extent[d], loc[d], -1.0).cpu().numpy() for d in (2, 1, 0)], indexing="ij")
        a, b, e = ((x, y, z), (y, z, x), (z, x, y))[c]
        v = -2 * scale * np.sin(math.pi * a) * (_mms_f(b, e) * math.pi ** 2 - _mms_p(b, e))
        v += 4.0 * np.cos(0.5 * math.pi * a) * np.sin(0.5 * math.pi * b + 0.3)  # drives pressure and shear too
        g.append(v.astype(DTYPES[case["dtype"]][1]).astype(np.float64))
    return {"nd": 3, "n": n, "extent": extent, "steps": _pt_steps(extent, n), "gravity": g,
            "bcs": (("slip", "slip"),) * 3, "glen": None, "eta": None}


def _plane(case, seed):
    n = (case["nx"], case["ny"])
    npd = DTYPES[case["dtype"]][1]
    rs = np.random.RandomState((seed + 77) % (1 << 31))
    if case["kind"] == "mms":
        scale, extent = float(rs.uniform(0.5, 2.0)), (1.0, 1.0)
        g = []
        for c in range(2):
            loc = (1, 0) if c == 0 else (0, 1)
            y, x = np.meshgrid(*[_coord(n[d], 1.0, loc[d]).cpu().numpy() for d in (1, 0)], indexing="ij")
            f = np.sin(math.pi * x) * np.cos(math.pi * y) if c == 0 else -np.cos(math.pi * x) * np.sin(math.pi * y)
            f = -2 * scale * math.pi ** 2 * f + 4.0 * np.cos(0.5 * math.pi * (x, y)[c]) * np.sin(math.pi * (y, x)[c] + 0.3)
            g.append(f.astype(npd).astype(np.float64))  # the second term drives pressure and shear too
        return {"nd": 2, "n": n, "extent": extent, "steps": _pt_steps(extent, n), "gravity": g,
                "bcs": (("slip", "slip"),) * 2, "glen": None, "eta": None}
    extent = (2.0, 1.0)
    return {"nd": 2, "n": n, "extent": extent, "steps": _pt_steps(extent, n), "gravity": (0.17, 1.0),
            "bcs": (("slip", "slip"), ("velocity", "traction")), "glen": (1.0, 2.0),
            "eta": _rounded(torch.exp(_smooth(rs, n, extent, (0, 0), 0.2)), case["dtype"])}


def _start2(case, seed, extent):
    n = (case["nx"], case["ny"])
    rs = np.random.RandomState(seed % (1 << 31))
    for f in F2:
        yield f, _rounded(_smooth(rs, n, extent, LOC[f], 0.05 if f[0] == "V" else 0.2), case["dtype"])


def _ice(n, seed, dtype):
    """Volume fractions of ice between a bed of 64 Gaussian bumps and a wavy surface on
    the unit cube: {group: {location: (n+3)^3 halo box}}, group "na" below the
    surface, "ns" above the bed; nonzero at indices 1..n+1 as the level-set path
    fills them."""
    dev = _device()
    rs = np.random.RandomState(seed % (1 << 31))
    a, w, cx, cy = (torch.tensor(v, device=dev) for v in (rs.uniform(0, 0.2, 64), rs.uniform(0.05, 0.2, 64),
                                                         rs.uniform(0, 1, 64), rs.uniform(0, 1, 64)))
    out = {"na": {}, "ns": {}}

    def at(d, vertex):
        h = 1.0 / n[d]
        return h * (torch.arange(n[d] + 1, dtype=torch.float64, device=dev) + (0.0 if vertex else 0.5))

    for name in ("ccc", "vvv", "vcc", "cvc", "ccv", "vvc", "vcv", "cvv"):
        x, y, z = (at(d, name[d] == "v") for d in range(3))
        ex = torch.exp(-((x[None] - cx[:, None]) / w[:, None]) ** 2)
        ey = torch.exp(-((y[None] - cy[:, None]) / w[:, None]) ** 2)
        bed = torch.einsum("b,by,bx->yx", a, ey, ex)
        surf = (0.6 + 0.05 * torch.sin(2 * math.pi * x))[None].expand_as(bed)
        hz = 1.0 / n[2]
        for group, v in (("na", (surf[None] - (z - 0.5 * hz)[:, None, None]) / hz),
                         ("ns", ((z + 0.5 * hz)[:, None, None] - bed[None]) / hz)):
            box = torch.zeros(tuple(m + 3 for m in reversed(n)), dtype=DTYPES[dtype][0], device=dev)
            box[1:n[2] + 2, 1:n[1] + 2, 1:n[0] + 2] = v.clamp_(0.0, 1.0).to(box.dtype)
            out[group][name] = box
    return out


def _inclusion_viscosity(n, rs, dtype):
    """Matrix of viscosity 1 with 1-16 circles of contrasting viscosity, smoothed in log
    space over a few cells; and the factor by which the velocity step has to shrink."""
    y, x = torch.meshgrid(*[(torch.arange(m, dtype=torch.float64, device=_device()) + 0.5) / m for m in (n[1], n[0])],
                          indexing="ij")
    lg = torch.zeros_like(x)
    for _ in range(int(rs.randint(1, 17))):
        r, cx, cy = float(rs.uniform(0.02, 0.15)), float(rs.uniform()), float(rs.uniform())
        v = float(np.clip(rs.normal(0.0, 3.0), -math.log(1e4), math.log(1e4)))
        lg[(x - cx) ** 2 + (y - cy) ** 2 <= r * r] = v
    edge = torch.nn.functional.pad
    for _ in range(4):
        p = edge(lg[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
        lg = 0.2 * (p[1:-1, 1:-1] + p[:-2, 1:-1] + p[2:, 1:-1] + p[1:-1, :-2] + p[1:-1, 2:])
    eta = _rounded(torch.exp(lg), dtype)
    p = edge(eta[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    v = 0.25 * (p[:-1, :-1] + p[:-1, 1:] + p[1:, :-1] + p[1:, 1:])
    ratio = 1.0
    for faces, cells, verts in ((0.5 * (p[1:-1, :-1] + p[1:-1, 1:]), torch.maximum(p[1:-1, :-1], p[1:-1, 1:]),
                                 torch.maximum(v[:-1], v[1:])),
                                (0.5 * (p[:-1, 1:-1] + p[1:, 1:-1]), torch.maximum(p[:-1, 1:-1], p[1:, 1:-1]),
                                 torch.maximum(v[:, :-1], v[:, 1:]))):
        ratio = max(ratio, float((torch.maximum(cells, verts) / faces).max()))
    return eta, ratio


def _inclusion(n, rs, dtype):
    eta, ratio = _inclusion_viscosity(n, rs, dtype)
    return {"nd": 2, "n": n, "extent": (1.0, 1.0), "steps": _pt_steps((1.0, 1.0), n, factor=1.1 * ratio),
            "gravity": (0.0, 0.0), "bcs": (("slip", "slip"),) * 2, "glen": None, "eta": eta,
            "wall": {(0, 1): (-1.0, 0.0), (1, 1): (0.0, 1.0)}}


def _glacier(n, seed, dtype):
    """Traction-free box, unit weight, unit viscosity, the glacier driver's steps."""
    return {"nd": 3, "n": n, "extent": (1.0, 1.0, 1.0), "gravity": (0.0, 0.0, 1.0), "glen": None, "eta": None,
            "steps": _pt_steps((1.0, 1.0, 1.0), n, r=0.9, re=5 * math.pi), "bcs": (("traction", "traction"),) * 3,
            "ice": _ice(n, seed, dtype)}


def _heat(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    rs = np.random.RandomState(seed % (1 << 31))
    h, lam, dt = [1.0 / m for m in n], 1.0, 1.0
    cfl = 0.99 / math.sqrt(3)
    re = math.pi + math.sqrt(math.pi ** 2 + 1.0 / lam / dt)
    theta, beta = 1.0 / re / cfl / min(h), (re * lam) / (cfl * min(h))
    T = _rounded(_smooth(rs, n, (1.0, 1.0, 1.0), (0, 0, 0), 1.0), case["dtype"])
    return {"n": n, "lam": lam, "dt": dt, "dtau_T": 1.0 / (dt + beta), "dtau_q": 1.0 / (1.0 + theta), "T": T,
            "value": {(1, 0): -0.1, (1, 1): 0.3}}  # fixed temperature on south and north, insulated elsewhere


# ---- the framework's side ------------------------------------------------------------
class _Memory:
    """A model's field storage for torch (keeps the model alive)."""

    def __init__(self, model, ptr, shape, strides, typestr):
        self.model = model
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides, "typestr": typestr,
                                         "version": 3}


class _Fields:
    """In-place views of a model's fields, one per buffer the model has shown."""

    def __init__(self, model, names):
        self.model, self.names, self.seen = model, names, {}
        g = model.grid
        self.esz = DTYPES[model.dtype][2]
        self.n, self.nd = g.dims, g.ndims
        self.pitch, self.rows, _ = model.layout()

    def box(self, name):
        """The whole halo box of a field."""
        m, s = self.model, (self.pitch * self.rows * self.esz, self.pitch * self.esz, self.esz)
        shape = tuple(v + 3 for v in reversed(self.n))
        mem = _Memory(m, m.device_ptr(name), shape, s[3 - self.nd:], "<f%d" % self.esz)
        return torch.as_tensor(mem, device="cuda")

    def interior(self, name):
        return self.box(name)[tuple(slice(1, 1 + s) for s in self.model.field_shape(name))]

    def now(self):
        out = {}
        for name in self.names:
            key = (name, self.model.device_ptr(name))
            if key not in self.seen:
                self.seen[key] = self.interior(name)
            out[name] = self.seen[key]
        return out


def _bc(fi, kind, nd, c=(0.0, 0.0, 0.0)):
    return {"periodic": fi.PBC, "slip": fi.SBC, "traction": fi.TBC, "velocity": fi.VBC}[kind](*(() if kind == "periodic" else c[:nd]))


def _model(pr, dtype):
    fi = _package()
    nd, n = pr["nd"], pr["n"]
    grid = fi.UniformGrid(origin=(0.0,) * nd, extent=pr["extent"], dims=n)
    wall = pr.get("wall", {})
    bcs = {k: tuple(_bc(fi, pr["bcs"][d][s], nd, wall.get((d, s), (0.0,) * nd)) for s in range(2))
           for d, k in enumerate("xyz"[:nd])}
    gravity = {k: (g if isinstance(g, float) else fi.ArrayField(g)) for k, g in zip("xyz", pr["gravity"])}
    if pr["glen"]:
        rheology = fi.ViscoplasticRegularisation(fi.PowerLawRheology(pr["glen"][0], 3), pr["glen"][1])
    else:
        rheology = fi.LinearViscousRheology(1.0 if pr["eta"] is None else fi.ArrayField(pr["eta"].cpu().numpy()))
    cls = fi.IsothermalImmersedBoundaryFullStokesModel if "ice" in pr else fi.IsothermalFullStokesModel
    m = cls(grid=grid, boundary_conditions=bcs, gravity=gravity, rheology=rheology, solver_params=pr["steps"], dtype=dtype)
    view = _Fields(m, ("eta", "eta_next"))
    for f in ("eta", "eta_next"):
        if pr["eta"] is None:
            view.interior(f).fill_(1.0)
        else:
            view.interior(f).copy_(pr["eta"])
    for group, boxes in pr.get("ice", {}).items():
        for name, box in boxes.items():
            view.box("%s_%s" % (group, name)).copy_(box)
    return m


_HOST = {}  # pinned host buffers of the program, by size and type


def _host(name, shape, dtype):
    """Pinned host memory that a program reads its results into."""
    key = (name, tuple(shape), dtype)
    if key not in _HOST:
        _HOST[key] = torch.empty(tuple(shape), dtype=DTYPES[dtype][0], pin_memory=torch.cuda.is_available()).numpy()
    return _HOST[key]


def prepare(case, seed):
    fam, dtype = case["family"], case["dtype"]
    gc.collect()  # models that the program has let go of give their memory back
    if torch.cuda.is_available():
        torch.cuda.empty_cache()
    if len(_HOST) > 24:
        _HOST.clear()
    if fam in ("slab", "mms3d", "plane"):
        pr = {"slab": _slab, "mms3d": _mms3d, "plane": _plane}[fam](case, seed)
        m = _model(pr, dtype)
        view = _Fields(m, (F3 if pr["nd"] == 3 else F2) + ("eta",))
        start = _start2(case, seed, pr["extent"]) if fam == "plane" else _start3(case, seed, pr["extent"], *_SCALES[fam])
        for f, v in start:
            view.interior(f).copy_(v)
        torch.cuda.synchronize()
        m.apply_bcs()
        return {"case": case, "model": m, "view": view}
    if fam == "glacier":
        n = (case["nx"], case["ny"], case["nz"])
        m = _model(_glacier(n, seed, dtype), dtype)
        torch.cuda.synchronize()
        m.apply_bcs()
        return {"case": case, "model": m, "host": {f: _host(f, m.field_shape(f), dtype) for f in ("P", "Vx", "Vy", "Vz")}}
    if fam == "inclusions":
        rs = np.random.RandomState(seed % (1 << 31))
        models = [_model(_inclusion(n, rs, dtype), dtype) for n in _members(case)]
        torch.cuda.synchronize()
        for m in models:
            m.apply_bcs()
        return {"case": case, "models": models, "batch": _package().BatchedStokes2D(models),
                "views": [_Fields(m, F2) for m in models]}
    if fam == "glaciers":
        models = [_model(_glacier((a, a, a), seed + 1000 * q, dtype), dtype) for q, (a,) in enumerate(_members(case))]
        torch.cuda.synchronize()
        for m in models:
            m.apply_bcs()
        host, parts = {}, {}
        for f in F3:
            sizes = [int(np.prod(m.field_shape(f))) for m in models]
            host[f] = _host(f, (sum(sizes),), dtype)
            at = np.cumsum([0] + sizes)
            parts[f] = [host[f][at[q]:at[q + 1]].reshape(m.field_shape(f)) for q, m in enumerate(models)]
        return {"case": case, "models": models, "batch": _package().BatchedIB3D(models), "host": host, "parts": parts}
    fi = _package()
    pr = _heat(case, seed)
    sides = (("west", "east"), ("south", "north"), ("bottom", "top"))
    bcs = {sides[d][s]: fi.heat.Value(pr["value"][d, s]) if (d, s) in pr["value"] else fi.heat.Flux(0.0)
           for d in range(3) for s in range(2)}
    m = fi.HeatDiffusionModel(grid=fi.UniformGrid(origin=(0.0,) * 3, extent=(1.0,) * 3, dims=pr["n"]),
                              boundary_conditions=bcs, physics={"λ_ρCp": pr["lam"]},
                              iter_params={"Δτ": {"T": pr["dtau_T"], "q": pr["dtau_q"]}}, dtype=dtype)
    T = pr["T"].cpu().numpy()
    m.set_field("T", T)
    m.set_field("T_o", T)
    m.apply_bcs()
    return {"case": case, "model": m, "dt": pr["dt"]}


_SCALES = {"slab": (1e-7, 3e-3, 1e-2), "mms3d": (0.5, 1.0, 1.0)}  # V, stresses, P of a state mid-solve


def run(state):
    case = state["case"]
    fam = case["family"]
    if fam in ("slab", "mms3d", "plane"):
        m = state["model"]
        norms = []
        for _ in range(case["rounds"]):
            m.advance(case["iters"])
            if case["norms"]:
                norms.append(m.residual_norms())
        return {"fields": state["view"].now(), "norms": norms}
    if fam == "glacier":
        m = state["model"]
        norms = []
        for _ in range(case["rounds"]):
            m.advance(case["iters"])
            norms.append(m.residual_norms())
        return {"fields": {f: m.get_field(f, out=a) for f, a in state["host"].items()}, "norms": norms}
    if fam == "inclusions":
        # one check-to-check round of a solve that is far from done
        items, _ = state["batch"].step(max_iter=1 << 30, ncheck=case["iters"], tol=1e-30, rounds=1)
        now = [v.now() for v in state["views"]]
        return {"fields": {f: torch.cat([v[f].reshape(-1) for v in now]) for f in F2},
                "measures": np.array([i["measure"] for i in items])}
    if fam == "glaciers":
        state["batch"].advance(case["iters"])
        state["batch"].synchronize()
        for f in F3:
            for m, a in zip(state["models"], state["parts"][f]):
                m.get_field(f, out=a)
        return {"fields": dict(state["host"])}
    state["model"].advance(case["iters"], state["dt"])
    return {"T": state["model"].get_field("T")}


# ---- the same pass in 64 bits ----------------------------------------------------------
class _Exact:
    """The staggered pseudo-transient iteration on halo boxes (index 0 and n+1.. ghosts),
    2D or 3D, in 64-bit torch."""

    def __init__(self, pr):
        self.pr, self.nd, self.n = pr, pr["nd"], pr["n"]
        self.names = F3 if self.nd == 3 else F2
        self.dev = _device()
        shape = tuple(m + 3 for m in reversed(self.n))
        self.a = {f: torch.zeros(shape, dtype=torch.float64, device=self.dev) for f in self.names}
        self.idx = [m / e for m, e in zip(self.n, pr["extent"])]
        s = pr["steps"]["Δτ"]
        self.dP, self.dT, self.dV = s["Pr"], s["τ"], s["V"]
        self.eta = torch.zeros(shape, dtype=torch.float64, device=self.dev)
        self.inner(self.eta, (0, 0, 0)).copy_(pr["eta"] if pr["eta"] is not None else torch.ones((), dtype=torch.float64))
        self.eta_faces(self.eta)
        self.g = []
        for c, g in enumerate(pr["gravity"]):
            if not isinstance(g, float):
                box = torch.zeros(shape, dtype=torch.float64, device=self.dev)
                self.inner(box, tuple(int(d == c) for d in range(3))).copy_(torch.as_tensor(g))
                g = self.at(box)
            self.g.append(g)
        self.ice = None
        if "ice" in pr:
            self.ice = {k: {q: b.to(torch.float64) for q, b in v.items()} for k, v in pr["ice"].items()}
            self.activity()

    # views of a box: the vertex range 1..n+1 of every dimension, moved by `by` (x, y, z)
    def at(self, box, **by):
        return box[tuple(slice(1 + by.get(k, 0), self.n[d] + 2 + by.get(k, 0)) for d, k in reversed(list(enumerate("xyz"[:self.nd]))))]

    def inner(self, box, loc):
        return box[tuple(slice(1, self.n[d] + 1 + loc[d]) for d in reversed(range(self.nd)))]

    def face(self, box, d, index, loc):
        """One layer along d: earlier dimensions over their whole storage, later ones over the interior."""
        s = [slice(None) if e < d else slice(1, self.n[e] + 1 + loc[e]) for e in range(self.nd)]
        s[d] = index
        return box[tuple(reversed(s))]

    def wrap(self, f, box, d):
        loc, n = LOC[f], self.n[d]
        F = lambda i: self.face(box, d, i, loc)  # noqa: E731
        if loc[d]:
            F(n + 1).copy_(F(1))
            F(0).copy_(F(n))
            F(n + 2).copy_(F(2))
        else:
            F(0).copy_(F(n))
            F(n + 1).copy_(F(1))

    def fixed(self, f, box, d, side, v):
        """Dirichlet value: the node itself, or the ghost that puts it on the face."""
        loc, n = LOC[f], self.n[d]
        F = lambda i: self.face(box, d, i, loc)  # noqa: E731
        if loc[d]:
            F(1 if side == 0 else n + 1).fill_(v)
        else:
            F(0 if side == 0 else n + 1).copy_(2.0 * v - F(1 if side == 0 else n))

    def value(self, d, side, c):
        return self.pr.get("wall", {}).get((d, side), (0.0, 0.0, 0.0))[c]

    def eta_faces(self, eta):
        for d in range(self.nd):
            if self.pr["bcs"][d][0] == "periodic":
                self.wrap("eta", eta, d)
                continue
            F = lambda i: self.face(eta, d, i, (0, 0, 0))  # noqa: E731
            F(0).copy_(F(1))
            F(self.n[d] + 1).copy_(F(self.n[d]))

    def stress_faces(self):
        shear = {0: (("txy", 1), ("txz", 2)), 1: (("txy", 0), ("tyz", 2)), 2: (("txz", 0), ("tyz", 1))}
        for d in range(self.nd):
            if self.pr["bcs"][d][0] == "periodic":
                for f in self.names:
                    if f[0] != "V":
                        self.wrap(f, self.a[f], d)
                continue
            for side in range(2):
                kind = self.pr["bcs"][d][side]
                if kind == "velocity":
                    continue
                if kind == "traction":
                    for f in ("P", ("txx", "tyy", "tzz")[d]):
                        self.fixed(f, self.a[f], d, side, self.value(d, side, d))
                for f, c in shear[d]:
                    if f in self.a:
                        self.fixed(f, self.a[f], d, side, self.value(d, side, c))

    def velocity_faces(self, eta):
        V = ("Vx", "Vy", "Vz")[:self.nd]
        for d in range(self.nd):
            if self.pr["bcs"][d][0] == "periodic":
                for f in V:
                    self.wrap(f, self.a[f], d)
                continue
            for side in range(2):
                kind = self.pr["bcs"][d][side]
                if kind == "velocity":
                    for c, f in enumerate(V):
                        self.fixed(f, self.a[f], d, side, self.value(d, side, c))
                elif kind == "slip":
                    self.fixed(V[d], self.a[V[d]], d, side, self.value(d, side, d))
        self.eta_faces(eta)

    def set(self, f, values):
        self.inner(self.a[f], LOC[f]).copy_(values)

    def begin(self):
        """The ghost fill that drivers do before iterating."""
        self.stress_faces()
        self.velocity_faces(self.eta)

    def activity(self):
        """Where the masked updates act: a point is empty below a fraction of 1e-6, and not
        valid next to an empty neighbour of its stencil."""
        na, ns = ({k: b < 1e-6 for k, b in self.ice[g].items()} for g in ("na", "ns"))
        at = self.at

        def near(w, loc):
            low = {"ccc": ("vcc", "cvc", "ccv"), "vcc": ("ccc", "vvc", "vcv"), "cvc": ("vvc", "ccc", "cvv"),
                   "ccv": ("vcv", "cvv", "ccc"), "vvc": ("cvc", "vcc", None), "vcv": ("ccv", None, "vcc"),
                   "cvv": (None, "ccv", "cvc")}[loc]
            bad = at(w[loc]).clone()
            for d, k in enumerate("xyz"):
                if low[d] is not None:  # a vertex looks back along d, a centre ahead
                    bad |= at(w[low[d]]) | at(w[low[d]], **{k: -1 if loc[d] == "v" else 1})
            return bad

        self.on = {q: ~(near(na, q) | at(ns[q])) for q in ("ccc", "vvc", "vcv", "cvv")}
        self.on.update({q: ~(near(ns, q) | at(na[q])) for q in ("vcc", "cvc", "ccv")})

    def step(self):
        A, at, dP, dT, dV = self.a, self.at, self.dP, self.dT, self.dV
        nd, (ix, iy), iz = self.nd, self.idx[:2], self.idx[2] if self.nd == 3 else 0.0
        ice, eta = self.ice, self.eta
        U = {f: A[f] for f in ("Vx", "Vy", "Vz")[:nd]}
        if ice:
            U = {f: A[f] * ice["ns"][q] for f, q in (("Vx", "vcc"), ("Vy", "cvc"), ("Vz", "ccv"))}

        def put(f, v, loc):
            at(A[f]).copy_(torch.where(self.on[loc], v, 0.0) if ice else v)

        exx = (at(U["Vx"], x=1) - at(U["Vx"])) * ix
        eyy = (at(U["Vy"], y=1) - at(U["Vy"])) * iy
        ezz = (at(U["Vz"], z=1) - at(U["Vz"])) * iz if nd == 3 else None
        div = exx + eyy if nd == 2 else exx + eyy + ezz
        e = at(eta)
        put("P", at(A["P"]) - div * e * dP, "ccc")
        for f, s in (("txx", exx), ("tyy", eyy), ("tzz", ezz))[:nd]:
            t = at(A[f])
            put(f, t - (t - 2.0 * e * (s - div / 3.0)) * dT[f[1:]], "ccc")
        del exx, eyy, ezz, div
        for f, p, q, (k, ik), (m, im), loc in (("txy", "Vy", "Vx", ("x", ix), ("y", iy), "vvc"),
                                               ("txz", "Vz", "Vx", ("x", ix), ("z", iz), "vcv"),
                                               ("tyz", "Vz", "Vy", ("y", iy), ("z", iz), "cvv"))[:1 if nd == 2 else 3]:
            s = 0.5 * ((at(U[p]) - at(U[p], **{k: -1})) * ik + (at(U[q]) - at(U[q], **{m: -1})) * im)
            ev = 0.25 * (e + at(eta, **{k: -1}) + at(eta, **{m: -1}) + at(eta, **{k: -1, m: -1}))
            t = at(A[f])
            put(f, t - (t - 2.0 * ev * s) * dT[f[1:]], loc)
        del U
        self.stress_faces()
        S = {f: A[f] for f in self.names if f[0] != "V"}
        if ice:
            S = {f: A[f] * ice["na"][{"txy": "vvc", "txz": "vcv", "tyz": "cvv"}.get(f, "ccc")] for f in S}
        dims = (("x", ix), ("y", iy), ("z", iz))[:nd]
        for c, (k, ik) in enumerate(dims):
            f, d = ("Vx", "Vy", "Vz")[c], ("txx", "tyy", "tzz")[c]
            r = (at(S[d]) - at(S[d], **{k: -1}) - (at(S["P"]) - at(S["P"], **{k: -1}))) * ik - self.g[c]
            for m, im in dims:
                if m != k:
                    t = S["t" + "".join(sorted(k + m))]
                    r = r + (at(t, **{m: 1}) - at(t)) * im
            r = r / (0.5 * (e + at(eta, **{k: -1})))
            if ice:
                loc = ("vcc", "cvc", "ccv")[c]
                r = r / at(ice["ns"][loc]).clamp(min=1e-6)
                put(f, at(A[f]) + r * dV[k], loc)
            else:
                at(A[f]).add_(r, alpha=dV[k])
        if self.pr["glen"]:
            def mean(t, k, m):
                return 0.25 * (at(t) + at(t, **{k: 1}) + at(t, **{m: 1}) + at(t, **{k: 1, m: 1}))

            s2 = 0.5 * sum(at(A[f]) ** 2 for f in ("txx", "tyy", "tzz")[:nd]) + mean(A["txy"], "x", "y") ** 2
            if nd == 3:
                s2 = s2 + mean(A["txz"], "x", "z") ** 2 + mean(A["tyz"], "y", "z") ** 2
            new = torch.zeros_like(eta)
            at(new).copy_(1.0 / (2.0 * self.pr["glen"][0] * s2 + 1.0 / self.pr["glen"][1]))
            self.eta = new
        self.velocity_faces(self.eta)

    def norms(self):
        """Largest and root-sum-square residuals of r_P and r_V, and the largest velocities."""
        A, at, ice = self.a, self.at, self.ice
        U, S = A, A
        if ice:
            U = {f: A[f] * ice["ns"][q] for f, q in (("Vx", "vcc"), ("Vy", "cvc"), ("Vz", "ccv"))}
            S = {f: A[f] * ice["na"][{"txy": "vvc", "txz": "vcv", "tyz": "cvv"}.get(f, "ccc")] for f in A if f[0] != "V"}
        out = [0.0] * 12
        dims = [(k, self.idx[d]) for d, k in enumerate("xyz"[:self.nd])]
        V = ("Vx", "Vy", "Vz")[:self.nd]

        def fold(q, r, loc, where):
            if ice:
                r = torch.where(self.on[where], r, 0.0)
            r = r[tuple(slice(0, self.n[d] + loc[d]) for d in reversed(range(self.nd)))]
            if q:
                for side, at_ in ((0, 0), (1, -1)):
                    if self.pr["bcs"][q - 1][side] in ("slip", "velocity"):
                        r = r.clone()
                        r.select(self.nd - q, at_).zero_()
            out[q], out[4 + q] = float(r.abs().max()), float(r.square().sum().sqrt())

        fold(0, sum((at(U[f], **{k: 1}) - at(U[f])) * ik for f, (k, ik) in zip(V, dims)), (0, 0, 0), "ccc")
        for c, (k, ik) in enumerate(dims):
            d = ("txx", "tyy", "tzz")[c]
            r = (at(S[d]) - at(S[d], **{k: -1}) - (at(S["P"]) - at(S["P"], **{k: -1}))) * ik - self.g[c]
            for m, im in dims:
                if m != k:
                    t = S["t" + "".join(sorted(k + m))]
                    r = r + (at(t, **{m: 1}) - at(t)) * im
            fold(c + 1, r, LOC[V[c]], ("vcc", "cvc", "ccv")[c])
            out[8 + c] = float(self.inner(A[V[c]], LOC[V[c]]).abs().max())
        return np.array(out)

    def fields(self, names):
        return {f: self.inner(self.eta if f == "eta" else self.a[f], LOC[f]) for f in names}


def exact(case, seed):
    fam, dtype = case["family"], case["dtype"]
    if fam in ("slab", "mms3d", "plane"):
        pr = {"slab": _slab, "mms3d": _mms3d, "plane": _plane}[fam](case, seed)
        e = _Exact(pr)
        start = _start2(case, seed, pr["extent"]) if fam == "plane" else _start3(case, seed, pr["extent"], *_SCALES[fam])
        for f, v in start:
            e.set(f, v)
        e.begin()
        norms = []
        for _ in range(case["rounds"]):
            for _ in range(case["iters"]):
                e.step()
            if case["norms"]:
                norms.append(e.norms())
        return {"fields": e.fields(e.names + ("eta",)), "norms": norms}
    if fam == "glacier":
        e = _Exact(_glacier((case["nx"], case["ny"], case["nz"]), seed, dtype))
        e.begin()
        norms = []
        for _ in range(case["rounds"]):
            for _ in range(case["iters"]):
                e.step()
            norms.append(e.norms())
        return {"fields": e.fields(("P", "Vx", "Vy", "Vz")), "norms": norms}
    if fam == "inclusions":
        rs = np.random.RandomState(seed % (1 << 31))
        got = []
        for n in _members(case):
            e = _Exact(_inclusion(n, rs, dtype))
            e.begin()
            for _ in range(case["iters"]):
                e.step()
            got.append(e.fields(F2))
        # the measure of a check is taken on the stored state, so it has no value of its own here
        return {"fields": {f: torch.cat([g[f].reshape(-1) for g in got]) for f in F2}, "measures": None}
    if fam == "glaciers":
        got = []
        for q, (a,) in enumerate(_members(case)):
            e = _Exact(_glacier((a, a, a), seed + 1000 * q, dtype))
            e.begin()
            for _ in range(case["iters"]):
                e.step()
            got.append(e.fields(F3))
        return {"fields": {f: torch.cat([g[f].reshape(-1) for g in got]) for f in F3}}
    pr = _heat(case, seed)
    n = pr["n"]
    T = torch.zeros(tuple(m + 2 for m in reversed(n)), dtype=torch.float64, device=_device())
    inn = (slice(1, -1),) * 3
    T[inn] = pr["T"]
    old = pr["T"]
    q = [torch.zeros(tuple(n[e] + (e == d) for e in (2, 1, 0)), dtype=torch.float64, device=_device()) for d in range(3)]

    def ghosts():
        for (d, s), v in pr["value"].items():
            ax = 2 - d
            T.select(ax, 0 if s == 0 else -1).copy_(2.0 * v - T.select(ax, 1 if s == 0 else -2))

    ghosts()
    for _ in range(case["iters"]):
        new = None
        for d in range(3):
            ax = 2 - d
            line = T[tuple(slice(None) if e == ax else slice(1, -1) for e in range(3))]
            q[d].sub_((q[d] + torch.diff(line, dim=ax) * (pr["lam"] * n[d])) * pr["dtau_q"])
            for s in range(2):
                if (d, s) not in pr["value"]:
                    q[d].select(ax, 0 if s == 0 else -1).zero_()
            g = torch.diff(q[d], dim=ax) * n[d]
            new = g if new is None else new + g
        T[inn] -= ((T[inn] - old) / pr["dt"] + new) * pr["dtau_T"]
        ghosts()
    return {"T": T[inn]}
