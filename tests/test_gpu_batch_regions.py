"""Batches of 2D models advance several iterations per launch on overlapping regions: the
state, the iteration counts and the measures equal those of the one-iteration sweeps bit for
bit (no-FMA and production builds), over members whose sides are multiples of the tiles or
not, odd and even numbers of iterations, retiring and joining members, a written state, and
more members than one launch takes."""
import numpy as np
import pytest

from conftest import load_fastice
from helpers import Pair

pytestmark = pytest.mark.gpu

TRAC, SLIP = ("traction", (0.1, -0.2)), ("slip", (0.05, -0.1))
VEL, VEL2 = ("velocity", (0.1, 0.2)), ("velocity", (-0.2, 0.3))
BCS = [((VEL, VEL2), (VEL2, VEL)), ((SLIP, VEL), (VEL2, TRAC)), ((TRAC, TRAC), (SLIP, SLIP))]
SIZES = [(24, 48), (25, 7), (130, 67), (3, 4), (23, 72)]
F2 = ("P", "txx", "tyy", "txy", "Vx", "Vy", "eta")


def _members(sizes, dtype, library):
    out = []
    for q, n in enumerate(sizes):
        p = Pair(n, BCS[q % 3], dtype=dtype, library=library, seed=50 + q, gravity=(0.3, -0.7, 0.0))
        out.append(p.model)
    return out


def _run(fi, models, plain):
    b = fi.BatchedStokes2D(models[:-1])
    if plain:
        b.set_variant(0)
    for k in (8, 3, 1, 2, 7):
        b.advance(k)
    models[1].set_field("Vx", 0.5 * models[1].get_field("Vx"))
    b.add(models[-1])
    first, _ = b.step(max_iter=1 << 30, ncheck=10, tol=1e-30, rounds=2)
    b.advance(1)  # the buffers trade roles before the captured round runs again
    models[0].advance(3)
    second, _ = b.step(max_iter=1 << 30, ncheck=10, tol=1e-30, rounds=1)
    b.remove(models[2])
    third, _ = b.step(max_iter=44, ncheck=4, tol=0.5, rounds=3)
    b.close()
    return [(i["iterations"], i["measure"]) for part in (first, second, third) for i in part]


@pytest.mark.parametrize("library", ["strict", "fast"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_regions_equal_sweeps(dtype, library):
    fi = load_fastice()
    a, c = _members(SIZES, dtype, library), _members(SIZES, dtype, library)
    got, want = _run(fi, a, False), _run(fi, c, True)
    bad = [(q, f) for q, (x, y) in enumerate(zip(a, c)) for f in F2 if not np.array_equal(x.get_field(f), y.get_field(f))]
    finite = all(np.isfinite(x.get_field(f)).all() for x in c for f in F2)
    for m in a + c:
        m.close()
    assert finite
    assert not bad, bad
    assert got == want


def test_more_members_than_a_launch_takes():
    fi = load_fastice()
    sizes = [(5 + q % 7, 6 + q % 5) for q in range(70)]
    a, c = _members(sizes, "f64", "strict"), _members(sizes, "f64", "strict")
    ba, bc = fi.BatchedStokes2D(a), fi.BatchedStokes2D(c)
    bc.set_variant(0)
    for b in (ba, bc):
        b.advance(6)
    want, _ = bc.step(max_iter=1 << 30, ncheck=6, tol=0.3, rounds=2)  # some of them retire
    got, _ = ba.step(max_iter=1 << 30, ncheck=6, tol=0.3, rounds=2)
    assert [(i["iterations"], i["measure"], i["status"]) for i in got] == [(i["iterations"], i["measure"], i["status"]) for i in want]
    for q in range(8):  # 62 left: one launch
        ba.remove(a[q])
        bc.remove(c[q])
    for b in (ba, bc):
        b.advance(9)
    for q in range(8, 70):
        ba.remove(a[q])
    ba.advance(4)  # no members: nothing moves
    bad = [(q, f) for q, (x, y) in enumerate(zip(a, c)) for f in F2 if not np.array_equal(x.get_field(f), y.get_field(f))]
    ba.close()
    bc.close()
    for m in a + c:
        m.close()
    assert not bad, bad
