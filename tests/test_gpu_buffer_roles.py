"""Launch tables and captured pairs of iterations name the buffers that held the state when they
were made.  A fused sweep, or a batched one of an odd number of iterations, leaves the state in
the other buffers: what was made before is made anew, bit for bit the same results (no-FMA
build) as models that never change buffers."""
import numpy as np
import pytest

from conftest import load_fastice
from helpers import make_bcs
from test_gpu_fusedib import BCS, _psi

pytestmark = pytest.mark.gpu

F2 = ("P", "txx", "tyy", "txy", "Vx", "Vy", "eta")
F3 = F2 + ("tzz", "txz", "tyz", "Vz")


def _fill(m, fields, seed):
    rng = np.random.default_rng(seed)
    for f in fields:
        v = 0.05 * rng.standard_normal(m.field_shape(f))
        m.set_field(f, 0.5 + np.abs(v) if f == "eta" else v)
    m.set_field("eta_next", m.get_field("eta"))
    m.apply_bcs()


def _glacier(fi, n, seed, path="auto", rheology=None):
    ext = tuple(0.05 * c for c in n)
    g = fi.UniformGrid(origin=(0.0, 0.0, 0.0), extent=ext, dims=n)
    m = fi.IsothermalImmersedBoundaryFullStokesModel(
        grid=g, boundary_conditions=make_bcs(fi, BCS["mixed"], 3), gravity={"x": 0.1, "y": 0.0, "z": 1.0},
        rheology=rheology or fi.LinearViscousRheology(1.3), solver_params=fi.pt_params(g), path=path, library="strict")
    for grp, psi in _psi(n, ext, "slab").items():
        m.omega_from_psi(grp, psi)
    _fill(m, F3, seed)
    return m


def _same(a, b, fields):
    return [f for f in fields if not np.array_equal(a.get_field(f), b.get_field(f))]


def test_shared_table_after_fused_sweeps():
    fi = load_fastice()
    sizes = [(24, 20, 12), (33, 9, 14)]
    members = [_glacier(fi, n, q) for q, n in enumerate(sizes)]
    plain = [_glacier(fi, n, q, path="reference") for q, n in enumerate(sizes)]
    b = fi.BatchedIB3D(members)
    b.advance(4)
    b.advance(3)  # too short for the fused sweep: shared launches in place
    b.advance(7)  # fused, odd: the other buffers hold the state
    b.synchronize()
    for m in members:
        m.set_field("Vx", 0.5 * m.get_field("Vx"))
    b.advance(3)
    b.advance(3)  # shared launches in place again
    b.advance(2)
    b.synchronize()
    for m in plain:
        m.advance(14)
        m.set_field("Vx", 0.5 * m.get_field("Vx"))
        m.advance(8)
    bad = [_same(x, y, F3) for x, y in zip(members, plain)]
    b.close()
    for m in members + plain:
        m.close()
    assert not any(bad), bad


def test_pairs_after_fused_sweeps():
    fi = load_fastice()
    glen = fi.ViscoplasticRegularisation(fi.PowerLawRheology(0.01, 3), 1.0)
    slow = fi.Relaxation(glen, 0.3)
    n = (24, 20, 12)
    out = []
    for path in ("auto", "reference"):
        m = _glacier(fi, n, 3, path=path, rheology=slow)
        m.advance(10)            # a moving viscosity runs in place, as captured pairs
        m.set_params(rheology=glen)
        m.advance(9)             # two full iterations, then seven fused ones
        m.set_params(rheology=slow)
        m.advance(1)
        m.advance(10)
        m.advance(10)
        out.append(m)
    bad = _same(*out, F3)
    for m in out:
        m.close()
    assert not bad, bad


def test_pairs_after_a_batch():
    fi = load_fastice()
    wall, top = ("velocity", (0.0, 0.0)), ("traction", (0.1, -0.2))
    g = fi.UniformGrid(origin=(0.0, 0.0), extent=(1.0, 1.25), dims=(40, 31))
    out = []
    for batched in (True, False):
        m = fi.IsothermalFullStokesModel(grid=g, boundary_conditions=make_bcs(fi, ((wall, wall), (wall, top)), 2),
                                         gravity={"x": 0.3, "y": -0.7}, rheology=fi.LinearViscousRheology(1.0),
                                         solver_params=fi.pt_params(g), path="reference", library="strict")
        _fill(m, F2, 5)
        m.set_field("eta", np.ones(m.field_shape("eta")))  # the viscosity of the law: held fixed by the batch
        m.set_field("eta_next", m.get_field("eta"))
        m.apply_bcs()
        m.advance(8)  # captured pairs
        if batched:
            with fi.BatchedStokes2D([m]) as b:
                b.advance(7)
        else:
            m.advance(7)
        m.advance(1)
        m.advance(8)
        m.advance(9)
        m.advance(8)
        out.append(m)
    bad = _same(*out, F2)
    for m in out:
        m.close()
    assert not bad, bad
