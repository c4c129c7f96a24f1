"""The fused 3D sweep at the edges of its tiles: sides that end a 32x8 tile exactly, one
short of it and one past it, so that a boundary's adjacent cell, its node and its ghost
fall into one tile or two, and z-blocks down to a single plane.  Bit for bit against the
CPU oracle in the no-FMA build, and the residual norms, which read the stress ghosts.
"""
import numpy as np
import pytest

from helpers import Pair

pytestmark = pytest.mark.gpu

TRAC = ("traction", (0.1, -0.2, 0.05))
TRAC2 = ("traction", (-0.3, 0.15, 0.2))
SLIP = ("slip", (0.05, -0.1, 0.2))
VEL = ("velocity", (0.1, 0.2, -0.3))
PER = ("periodic", ())
BCS = {
    "traction_box": ((TRAC, TRAC2), (TRAC2, TRAC), (TRAC, TRAC2)),
    "slip_traction": ((SLIP, TRAC), (TRAC, SLIP), (SLIP, TRAC)),
    "velocity_traction": ((TRAC, VEL), (VEL, TRAC), (TRAC, VEL)),
    "periodic_x": ((PER, PER), (TRAC, VEL), (VEL, SLIP)),
    "periodic_y": ((VEL, TRAC), (PER, PER), (TRAC, TRAC2)),
}


def zb_variant(lib, zb):
    names = [lib.fi_fused_variant_name(v).decode() for v in range(lib.fi_fused_variant_count())]
    return names.index(f"tile32x8_zb{zb}")


@pytest.mark.parametrize("bc", list(BCS))
@pytest.mark.parametrize("n", [(31, 7, 4), (32, 8, 3), (33, 9, 5), (64, 15, 8), (63, 16, 7)])
def test_tile_edges_bitwise(bc, n):
    p = Pair(n, BCS[bc], path="fused", library="strict", seed=21, rheo={"kind": "glen", "eta_reg": 10.0})
    for zb in (1, 2, 4, 32):
        p.model.set_variant(zb_variant(p.model.lib, zb))
        p.advance(2)
    bad = p.bitwise_equal()
    a, b = p.model.residual_norms(), p.oracle.residual_norms()
    p.close()
    assert not bad, bad
    np.testing.assert_array_equal(a[[0, 1, 2, 3, 8, 9, 10]], b[[0, 1, 2, 3, 8, 9, 10]])


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n", [(5, 4, 3), (96, 40, 33), (40, 30, 64)])
def test_default_shape_bitwise(dtype, n):
    p = Pair(n, BCS["slip_traction"], path="fused", library="strict", dtype=dtype, seed=22)
    p.advance(5)
    bad = p.bitwise_equal()
    p.close()
    assert not bad, bad
