"""2D models advance several iterations per launch, each CTA on a region whose edge layers
are thrown away: sides around the region and tile sizes, every kind of side, iteration
counts that split into launches of different depth, bit for bit against the CPU oracle in
the no-FMA build (so also against the reference-shaped path)."""
import numpy as np
import pytest

from helpers import Pair

pytestmark = pytest.mark.gpu

TRAC = ("traction", (0.1, -0.2))
TRAC2 = ("traction", (-0.3, 0.15))
SLIP = ("slip", (0.05, -0.1))
VEL = ("velocity", (0.1, 0.2))
VEL2 = ("velocity", (-0.2, 0.3))
PER = ("periodic", ())
BCS = {
    "velocity_box": ((VEL, VEL2), (VEL2, VEL)),
    "traction_box": ((TRAC, TRAC2), (TRAC2, TRAC)),
    "mixed": ((SLIP, VEL), (VEL2, TRAC)),
    "periodic_x": ((PER, PER), (VEL, TRAC)),
    "periodic": ((PER, PER), (PER, PER)),
}


@pytest.mark.parametrize("bc", list(BCS))
@pytest.mark.parametrize("n", [(3, 4), (23, 8), (24, 9), (25, 7), (57, 41), (130, 67)])
def test_bitwise(bc, n):
    p = Pair(n, BCS[bc], library="strict", seed=31, gravity=(0.3, -0.7, 0.0), rheo={"kind": "glen", "A": 0.01, "eta_reg": 1.0})
    for k in (2, 3, 5, 1, 9):
        p.advance(k)
    bad = p.bitwise_equal()
    prev, want = p.model.get_field("eta_next"), p.oracle.interior("eta_next")
    a, b = p.model.residual_norms(), p.oracle.residual_norms()
    p.close()
    assert not bad, bad
    assert np.array_equal(prev.view(np.uint64), want.view(np.uint64))
    assert np.isfinite(want).all()
    np.testing.assert_array_equal(a[[0, 1, 2, 8, 9]], b[[0, 1, 2, 8, 9]])


@pytest.mark.parametrize("rheo", [{"kind": "linear", "eta": 1.3}, {"kind": "relax_glen", "rate": 0.3, "scale": None}])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_rheologies_bitwise(rheo, dtype):
    p = Pair((66, 35), BCS["mixed"], library="strict", dtype=dtype, seed=32, gravity=(0.3, -0.7, 0.0), rheo=rheo)
    p.advance(13)
    bad = p.bitwise_equal()
    p.close()
    assert not bad, bad


def test_pointers_stay_current():
    # a state pointer taken before an advance still holds the current state after it
    p = Pair((40, 30), BCS["mixed"], seed=33)
    before = {f: p.model.device_ptr(f) for f in ("P", "Vx", "txy")}
    p.model.advance(11)
    assert {f: p.model.device_ptr(f) for f in before} == before
    p.close()
