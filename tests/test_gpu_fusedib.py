"""The fused sweep of 3D immersed-boundary models (the default path once two full iterations
have run) against the CPU oracle, bit for bit in the no-FMA build: box sizes at the edges of
its 32x8 columns, ice that touches every side or none, every kind of side, state written
between advances, a state pointer handed out, and members of a batch."""
import numpy as np
import pytest

from conftest import load_fastice
from helpers import Pair

pytestmark = pytest.mark.gpu

TRAC, TRAC2 = ("traction", (0.3, -0.1, 0.2)), ("traction", (0.0, 0.1, -0.2))
SLIP, SLIP2 = ("slip", (0.1, -0.1, 0.05)), ("slip", (0.0, 0.2, 0.0))
VEL, VEL2 = ("velocity", (0.1, -0.2, 0.05)), ("velocity", (-0.1, 0.1, 0.1))
BCS = {
    "traction_box": ((TRAC, TRAC2), (TRAC2, TRAC), (TRAC, TRAC2)),
    "velocity_box": ((VEL, VEL2), (VEL2, VEL), (VEL, VEL2)),
    "slip_box": ((SLIP, SLIP2), (SLIP2, SLIP), (SLIP, SLIP2)),
    "mixed": ((VEL, TRAC), (SLIP, TRAC2), (VEL2, TRAC)),
    "mixed2": ((TRAC, SLIP), (TRAC2, VEL), (TRAC, SLIP2)),
}
GLEN = {"kind": "glen", "A": 0.01, "eta_reg": 1.0}
LINEAR = {"kind": "linear", "eta": 1.3}


def _psi(n, ext, shape):
    x = [(np.arange(n[d] + 3) - 1) / n[d] for d in range(3)]
    Z, Y, X = np.meshgrid(x[2], x[1], x[0], indexing="ij")
    if shape == "full":  # ice everywhere
        return {"na": -np.ones_like(X), "ns": -np.ones_like(X)}
    if shape == "slab":  # a tilted layer on a tilted bed, cut by the sides
        return {"na": (Z - 0.75 + 0.4 * X - 0.1 * Y) * ext[2], "ns": -(Z - 0.3 + 0.2 * X) * ext[2]}
    ball = lambda c, r: np.sqrt(sum((ext[d] * (a - c[d])) ** 2 for d, a in enumerate((X, Y, Z)))) - r
    return {"na": ball((0.5, 0.5, 0.5), 0.35 * min(ext)), "ns": -ball((0.5, 0.5, -0.1), 0.45 * min(ext))}


def _pair(n, bc, shape, rheo=GLEN, dtype="f64", seed=41):
    ext = tuple(0.05 * c for c in n)
    return Pair(n, BCS[bc], rheo=rheo, library="strict", dtype=dtype, seed=seed, origin=(0.0, 0.0, 0.0), extent=ext,
                immersed_psi=_psi(n, ext, shape))


def _check(p):
    bad = p.bitwise_equal()
    finite = all(np.isfinite(p.oracle.interior(f)).all() for f in p.state)
    assert finite
    assert not bad, bad


@pytest.mark.parametrize("shape", ["full", "slab", "ball"])
@pytest.mark.parametrize("n", [(31, 7, 12), (32, 8, 9), (33, 9, 4), (66, 17, 35)])
@pytest.mark.parametrize("bc", list(BCS))
def test_bitwise(bc, n, shape):
    p = _pair(n, bc, shape)
    p.advance(9)
    _check(p)
    p.advance(1)  # an odd number in all: the other buffers hold the state
    p.advance(3)
    _check(p)
    a, b = p.model.residual_norms(), p.oracle.residual_norms()
    prev, want = p.model.get_field("eta_next"), p.oracle.interior("eta_next")
    p.close()
    np.testing.assert_array_equal(a[[0, 1, 2, 3]], b[[0, 1, 2, 3]])
    assert np.array_equal(prev.view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("rheo", [LINEAR, GLEN, {"kind": "relax_glen", "eta_reg": 1.0}], ids=["linear", "glen", "relaxed"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_written_state(dtype, rheo):
    # values everywhere, inactive points included; then few iterations, boundary values
    # put in again, a state pointer
    p = _pair((41, 13, 22), "mixed", "slab", rheo=rheo, dtype=dtype)
    p.advance(10)
    rng = np.random.default_rng(5)
    for name in ("P", "txy", "Vz", "eta"):
        v = 0.1 * rng.standard_normal(p.model.field_shape(name))
        v = (0.5 + np.abs(v) if name == "eta" else v).astype(np.float64 if dtype == "f64" else np.float32)
        p.model.set_field(name, v)
        p.oracle.set_interior(name, v)
    p.advance(3)
    _check(p)
    p.advance(7)
    p.model.apply_bcs()
    p.oracle.apply_initial_bcs()
    p.advance(2)
    p.advance(8)
    _check(p)
    at = p.model.device_ptr("Vx")
    p.advance(9)
    assert p.model.device_ptr("Vx") == at
    _check(p)
    p.close()


def test_moved_ice():
    # new fractions between advances: other columns hold ice
    from conftest import load_oracle
    O = load_oracle()
    n = (40, 20, 24)
    p = _pair(n, "mixed2", "ball")
    p.advance(9)
    ext = tuple(0.05 * c for c in n)
    dx = tuple(e / c for e, c in zip(ext, n))
    for grp, psi in _psi(n, ext, "slab").items():
        p.model.omega_from_psi(grp, psi)
        new = O.volfrac3d(n, dx, psi)
        for k, c in enumerate(O.MASK_COMPONENTS):
            p.oracle.masks[grp][k][...] = new[c]
    p.advance(11)
    _check(p)
    p.close()


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_batch_members(dtype):
    # shared sweeps over members of different sizes, odd and even numbers of iterations, a
    # member that advances alone between them
    fi = load_fastice()
    pairs = [_pair((33, 9, 14), "mixed", "slab", dtype=dtype), _pair((20, 30, 10), "mixed2", "ball", LINEAR, dtype=dtype),
             _pair((70, 12, 9), "traction_box", "full", dtype=dtype)]
    b = fi.BatchedIB3D([p.model for p in pairs])
    for k in (3, 7, 8, 2, 1):
        b.advance(k)
    b.synchronize()
    pairs[1].model.advance(9)
    pairs[1].model.synchronize()
    b.advance(6)
    b.synchronize()
    pairs[1].oracle.advance(9)
    for p in pairs:
        p.oracle.advance(27)
        _check(p)
    b.close()
    for p in pairs:
        p.close()
