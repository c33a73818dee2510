"""A claw call whose step limit is below one takes no step: nv(1) <= 0, or a
fixed dt that leads away from tend (nv(1) = (tend - tstart) / dt < 0)."""
import pytest

from classic_b200 import problems
from classic_b200.solver import BatchSolver, Solver
from helpers import same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu

GRIDS = {1: lambda: problems.acoustics_1d_config(mx=100), 2: lambda: problems.random_acoustics_2d(20, 17),
         3: lambda: problems.random_acoustics_3d(9, 8, 7)}
KEYS = ("t_reached", "dt_next", "dt_min", "steps_taken", "cfl_max_seen", "cfl_last")


@pytest.mark.parametrize("steps_max,dt,variable", [(0, 5e-4, True), (-2, 5e-4, True), (50, -5e-4, False)])
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_grid(dim, steps_max, dt, variable):
    rd, solver, params, q0, aux = GRIDS[dim]()
    rd.clawdata.steps_max, rd.clawdata.dt_variable = steps_max, variable
    g, o = Solver(rd.clawdata, solver, params), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        if aux is not None:
            s.set_aux(aux)
    (_, sg), (_, so) = g.advance(0.0, 0.05, dt), o.advance(0.0, 0.05, dt)
    assert so["steps_taken"] == 0
    for key in KEYS:
        assert sg[key] == so[key], key
    assert same(g.get_q(), q0)
    g.close()


def test_batch():
    probs = [problems.random_acoustics_2d(n, n) for n in (16, 21)]
    for p in probs:
        p[0].clawdata.steps_max = -2
    b = BatchSolver([p[0] for p in probs], probs[0][1], probs[0][2])
    for k, p in enumerate(probs):
        b.set_q(k, p[3])
    _, stats = b.advance(0.0, 0.05, 1e-3)
    for k, p in enumerate(probs):
        assert stats[k]["steps_taken"] == 0 and stats[k]["t_reached"] == 0.0
        assert same(b.get_q(k), p[3])
    b.close()
