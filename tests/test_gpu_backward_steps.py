"""Steps of negative dt (claw runs backward too): the Courant number is
|dt/dx| c whichever way time runs, where the kernels know it without a face
(constant speeds, the largest c of the medium) as where they fold it over faces."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import BatchSolver, Solver
from helpers import same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu

LIMITERS = ["minmod", "superbee", "vanleer", "mc", "none"]


def _step(prob, precision="fp64", **kw):
    rd, solver, params, q0, aux = prob
    g, o = Solver(rd.clawdata, solver, params, precision, **kw), OracleGrid(rd.clawdata, solver, params, **kw)
    for s in (g, o):
        s.set_q(q0)
        if aux is not None:
            s.set_aux(aux)
    dt = -0.4 * min(o.dxs) / 2.0
    cg, co = g.step(dt), o.step(dt)
    qg = g.get_q()
    g.close()
    return cg, co, qg, o.get_q()


@pytest.mark.parametrize("limiter", LIMITERS)
@pytest.mark.parametrize("split", ["unsplit", "godunov", "strang"])
@pytest.mark.parametrize("precision", ["fp64", "fp64_fma", "fp32"])
def test_acoustics_2d(precision, split, limiter):
    """c = 2: exact in FP32."""
    prob = problems.random_acoustics_2d(61, 37, seed=5, limiter=limiter)
    prob[0].clawdata.dimensional_split = split
    cg, co, qg, qo = _step(prob, precision)
    assert co > 0.0 and cg == co
    if precision == "fp64":
        assert same(qg, qo)


@pytest.mark.parametrize("precision", ["fp64", "fp64_fma", "fp32"])
@pytest.mark.parametrize("trans", [0, 22])
def test_acoustics_3d(trans, precision):
    """Media that FP32 holds exactly, so that the Courant number is the oracle's
    there too."""
    rd, solver, params, q0, aux = problems.random_acoustics_3d(19, 14, 11, seed=6, trans=trans)
    aux = np.float32(aux).astype(np.float64)
    cg, co, _, _ = _step((rd, solver, params, q0, aux), precision)
    assert co > 0.0 and cg == co


def test_advance():
    """A variable-dt call that starts backward: dt stays negative to the step limit."""
    rd, solver, params, q0, _ = problems.random_acoustics_2d(40, 30, seed=7)
    rd.clawdata.steps_max = 4
    g, o = Solver(rd.clawdata, solver, params), OracleGrid(rd.clawdata, solver, params)
    g.set_q(q0)
    o.set_q(q0)
    (ig, sg), (io, so) = g.advance(0.0, 0.05, -1e-3), o.advance(0.0, 0.05, -1e-3)
    assert ig == io == 11
    for key in ("t_reached", "dt_next", "steps_taken", "cfl_max_seen", "cfl_last", "dt_min"):
        assert sg[key] == so[key], key
    assert same(g.get_q(), o.get_q())
    g.close()


def test_batch():
    probs = [problems.random_acoustics_2d(n, n + 5, seed=n) for n in (20, 33)]
    for p in probs:
        p[0].clawdata.steps_max = 3
    b = BatchSolver([p[0] for p in probs], probs[0][1], probs[0][2])
    for k, p in enumerate(probs):
        b.set_q(k, p[3])
    info, stats = b.advance(0.0, 0.05, -1e-3)
    assert info == 11
    for k, (rd, solver, params, q0, _) in enumerate(probs):
        o = OracleGrid(rd.clawdata, solver, params)
        o.set_q(q0)
        _, so = o.advance(0.0, 0.05, -1e-3)
        assert stats[k]["cfl_last"] == so["cfl_last"] and stats[k]["dt_next"] == so["dt_next"]
        assert same(b.get_q(k), o.get_q())
    b.close()
