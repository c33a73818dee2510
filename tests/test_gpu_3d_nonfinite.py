"""A NaN or an infinity in one cell of a contracted or FP32 3D run: it reaches no
cell that it would not reach in the reference's order of operations (a wave whose
upwind neighbour's strength is NaN is limited to a finite one there too)."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64_fma", "fp32"])
@pytest.mark.parametrize("limiter", [[x, x] for x in ("minmod", "superbee", "vanleer", "mc")] +
                         [["minmod", "superbee"], ["mc", "vanleer"], ["superbee", "none"]])
@pytest.mark.parametrize("field,value", [(0, np.nan), (3, np.nan), (0, np.inf), (3, -np.inf)])
def test_spread(field, value, limiter, precision):
    rd, solver, params, q0, aux = problems.random_acoustics_3d(25, 20, 21, seed=11)
    rd.clawdata.limiter = limiter
    q0[field, 10, 9, 12] = value
    g, o = Solver(rd.clawdata, solver, params, precision), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        s.set_aux(aux)
    for _ in range(3):
        g.step(0.004)
        o.step(0.004)
    bad, ref = ~np.isfinite(g.get_q()), ~np.isfinite(o.get_q())
    g.close()
    assert ref.any() and bad.any()
    assert not (bad & ~ref).any(), (bad.sum(), ref.sum())
