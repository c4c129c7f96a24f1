"""A batch of more members than one launch takes, in which all members of one launch have
retired while others go on: state, iteration counts, measures and statuses equal those of the
one-iteration sweeps bit for bit, with the captured round and without it."""
import numpy as np
import pytest

from conftest import load_fastice
from helpers import make_bcs

pytestmark = pytest.mark.gpu

F2 = ("P", "txx", "tyy", "txy", "Vx", "Vy")
GROUP = 64  # members of a launch


def _model(fi, q, rest):
    """A random state under gravity, or (rest) one that solves its problem: zero."""
    n = (40 + 5 * (q % 9), 150 + q % 4) if q < 6 else (20 + q % 7, 30 + q % 5)
    grid = fi.UniformGrid(origin=(0.0, 0.0), extent=(1.0, 1.25), dims=n)
    wall = ("velocity", (0.0, 0.0))
    m = fi.IsothermalFullStokesModel(grid=grid, boundary_conditions=make_bcs(fi, ((wall, wall), (wall, ("traction", (0.0, 0.0)))), 2),
                                     gravity={"x": 0.0, "y": 0.0 if rest else 1.0}, rheology=fi.LinearViscousRheology(1.0),
                                     solver_params=fi.pt_params(grid))
    rng = np.random.default_rng(q)
    for f in F2:
        m.set_field(f, (0.0 if rest else 0.1) * rng.standard_normal(m.field_shape(f)))
    for f in ("eta", "eta_next"):
        m.set_field(f, np.ones(m.field_shape(f)))
    m.apply_bcs()
    return m


def _run(fi, plain, use_graph):
    late = range(2 * GROUP, 2 * GROUP + 2)
    models = [_model(fi, q, GROUP <= q < 2 * GROUP) for q in range(2 * GROUP + 2)]
    b = fi.BatchedStokes2D(models)
    if plain:
        b.set_variant(0)
    out, opts = [], dict(max_iter=1 << 30, ncheck=10, tol=1e-12, use_graph=use_graph)
    out += b.step(rounds=8, **opts)[0]  # the middle group retires in the first of them
    for q in late:  # the last group follows: members at rest take the place of its two
        b.remove(models[q])
        rest = _model(fi, q, True)
        models.append(rest)
        b.add(rest)
    out += b.step(rounds=12, **opts)[0]
    status = [i["status"] for i in out[-(2 * GROUP + 2):]]
    state = [m.get_field(f) for m in models for f in F2]
    b.close()
    for m in models:
        m.close()
    return [(i["iterations"], i["measure"], i["status"]) for i in out], status, state


@pytest.mark.parametrize("use_graph", [True, False], ids=["graph", "launches"])
def test_empty_groups(use_graph):
    fi = load_fastice()
    want, _, state_w = _run(fi, True, use_graph)
    got, status, state = _run(fi, False, use_graph)
    assert set(status[:GROUP]) == {"active"} and set(status[GROUP:]) == {"converged"}, status
    assert got == want
    assert all(np.array_equal(x, y) and np.isfinite(y).all() for x, y in zip(state, state_w))


@pytest.mark.parametrize("use_graph", [True, False], ids=["graph", "launches"])
def test_solve_again(use_graph):
    # launches follow the retirements; the next solve starts with all members again
    fi = load_fastice()
    out = []
    for plain in (True, False):
        models = [_model(fi, q, q % 3 == 1 or q > GROUP) for q in range(GROUP + 9)]
        b = fi.BatchedStokes2D(models)
        if plain:
            b.set_variant(0)
        items = []
        for tol in (5e-2, 2e-2, 1e-2):
            items += b.solve(max_iter=3000, ncheck=50, tol=tol, use_graph=use_graph)[0]
            for q in (2, 5, GROUP + 3):
                models[q].set_field("Vx", 0.3 + models[q].get_field("Vx"))
        out.append(([(i["iterations"], i["measure"], i["status"]) for i in items], [m.get_field(f) for m in models for f in F2]))
        b.close()
        for m in models:
            m.close()
    (want, state_w), (got, state) = out
    assert len({i[0] for i in want}) > 3  # members retire at several checks
    assert got == want
    assert all(np.array_equal(x, y) and np.isfinite(y).all() for x, y in zip(state, state_w))
