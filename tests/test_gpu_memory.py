"""Models on a device with little memory left.  The second state buffer of the default path of
2D and immersed-boundary models is taken if there is room and given back where an allocation
that the model cannot do without would fail: what fitted without it still runs, in place and
with the same bits (no-FMA build)."""
import gc

import numpy as np
import pytest
import torch

from conftest import load_fastice
from helpers import make_bcs

pytestmark = pytest.mark.gpu

MB = 1 << 20
F2 = ("P", "txx", "tyy", "txy", "Vx", "Vy", "eta")
TRAC, VEL = ("traction", (0.1, -0.2, 0.1)), ("velocity", (0.1, 0.2, 0.0))


class Fill:
    """Leaves `left` bytes of the device's memory free."""

    def __init__(self, left):
        gc.collect()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.t = torch.empty(max(free - left, 0), dtype=torch.uint8, device="cuda")
        free, _ = torch.cuda.mem_get_info()
        assert left - 64 * MB < free <= left + 64 * MB, free

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        del self.t
        torch.cuda.empty_cache()


def _model(fi, n, path="auto", dtype="f64"):
    nd = len(n)
    ext = tuple(1.0 + 0.25 * d for d in range(nd))
    g = fi.UniformGrid(origin=(0.0,) * nd, extent=ext, dims=n)
    cls = fi.IsothermalFullStokesModel if nd == 2 else fi.IsothermalImmersedBoundaryFullStokesModel
    bcs = tuple((VEL if d else TRAC, TRAC) for d in range(nd))
    m = cls(grid=g, boundary_conditions=make_bcs(fi, tuple((tuple((k, c[:nd]) for k, c in s)) for s in bcs), nd),
            gravity=dict(zip("xyz", (0.3, -0.7, 0.2)[:nd])), rheology=fi.LinearViscousRheology(1.0), solver_params=fi.pt_params(g),
            path=path, dtype=dtype, library="strict")
    if nd == 3:
        z = (np.arange(n[2] + 3) - 1) / n[2]
        psi = np.broadcast_to(z[:, None, None], tuple(c + 3 for c in n[::-1]))
        m.omega_from_psi("na", np.ascontiguousarray(psi - 0.8))
        m.omega_from_psi("ns", np.ascontiguousarray(0.2 - psi))
    x = np.linspace(0.0, 3.0, m.field_shape("P")[-1])
    m.set_field("P", np.broadcast_to(0.1 * np.sin(x), m.field_shape("P")).copy())
    for f in ("eta", "eta_next"):
        m.set_field(f, np.ones(m.field_shape(f)))
    m.apply_bcs()
    return m


def _want(fi, n, fields, steps):
    m = _model(fi, n, path="reference")
    for k in steps:
        m.advance(k)
    out = {f: m.get_field(f) for f in fields}
    m.close()
    return out


def test_plane_without_room_for_a_second_state():
    fi = load_fastice()
    n = (3000, 2500)
    field = 3040 * 2503 * 8
    want = _want(fi, n, F2, (5, 4))
    torch.zeros(1, device="cuda")
    with Fill(9 * field + 160 * MB):  # 8 fields and a staging buffer; 7 more do not fit
        m = _model(fi, n)
        m.advance(5)
        m.advance(4)
        bad = [f for f in F2 if not np.array_equal(m.get_field(f), want[f])]
        m.close()
    assert not bad, bad


def test_glacier_gives_its_second_state_back():
    fi = load_fastice()
    n = (190, 180, 170)
    field = 224 * 183 * 173 * 8
    fields = F2 + ("tzz", "txz", "tyz", "Vz")
    want = _want(fi, n, fields, (9, 8))
    m = _model(fi, n)
    m.advance(9)  # an odd number of fused sweeps: the state is in the second buffer
    m.synchronize()
    with Fill(2 * field + 32 * MB):  # the four residual fields do not fit beside it
        m.compute_residuals()
        r = m.get_field("rVz")
        free, _ = torch.cuda.mem_get_info()
        assert free > 6 * field  # ten fields back, four of them taken
        m.advance(8)
        bad = [f for f in fields if not np.array_equal(m.get_field(f), want[f])]
    m.close()
    assert np.isfinite(r).all() and np.abs(r).max() > 0
    assert not bad, bad


def test_mixed_solve_without_room_beside_the_second_states():
    fi = load_fastice()
    n = (2600, 2400)
    field = 2656 * 2403 * 8
    kw = dict(max_iter=400, ncheck=20, tol=1e-12, window=20, mode="mixed")
    out = []
    for left in (None, 12 * field):  # shadow 5.5 to 9 fields, residuals 3, the members' second states
        m = _model(fi, n)
        with fi.BatchedStokes2D([m]) as b:
            if left:
                with Fill(left):
                    items, _ = b.solve(**kw)
            else:
                items, _ = b.solve(**kw)
        out.append((items, [m.get_field(f) for f in F2]))
        m.close()
    assert out[0][0] == out[1][0] and out[0][0][0]["iterations"] > 60, out[0][0]  # two corrections and more
    assert all(np.array_equal(a, b) for a, b in zip(out[0][1], out[1][1]))


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_admission_estimates_cover_what_models_hold(dtype):
    fi = load_fastice()
    from fastice_b200 import scenarios, serving
    esz = 8 if dtype == "f64" else 4

    def free():
        gc.collect()  # (models that other tests left behind)
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def glacier(n):
        m = scenarios.bed_model(2, n, dtype=dtype)[0]
        m.advance(20)
        m.compute_residuals()
        m.residual_norms()
        return [m]

    def planes(n):
        ms = [scenarios.inclusion_model(s, n=n, dtype=dtype)[0] for s in range(4)]
        with fi.BatchedStokes2D(ms) as b:
            b.step(max_iter=100, ncheck=10, tol=1e-3, rounds=1)
        return ms

    for m in glacier(16) + planes((32, 32)):  # kernels and libraries load
        m.close()
    for make, n, want in [(glacier, n, serving.footprint_3d_ib((n,) * 3, esz)) for n in (32, 64, 96)] + \
                         [(planes, n, 4 * serving.footprint_2d(n, esz)) for n in ((128, 128), (511, 500), (1200, 900))]:
        before = free()
        ms = make(n)
        used = before - free()
        for m in ms:
            m.close()
        # (small allocations come in pieces of 2 MB)
        assert used <= want + (4 << 20) and want <= 1.35 * used + (4 << 20), (n, used, want)
