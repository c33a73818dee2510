"""Two 1D grids of one kernel alive at once: the one set up first needs more
shared memory than the one set up after it."""
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build,large,small", [
    (problems.acoustics_1d_config, 6000, 900),        # 192 KB, then 29 KB
    (problems.acoustics_1d_heterogeneous, 4000, 3100),
    (problems.euler_1d_wcblast, 4500, 600)])
def test_large_then_small(build, large, small):
    grids = []
    for mx in (large, small):
        rd, solver, params, q0, aux = build(mx=mx)
        s = Solver(rd, solver, params)
        s.set_q(q0)
        if aux is not None:
            s.set_aux(aux)
        grids.append((s, rd, solver, params, q0, aux))
    for s, rd, solver, params, q0, aux in grids:
        o = OracleGrid(rd.clawdata, solver, params)
        o.set_q(q0)
        if aux is not None:
            o.set_aux(aux)
        dt = 1e-6
        assert s.step(dt) == o.step(dt)
        assert same(s.get_q(), o.get_q())
    for g in grids:
        g[0].close()
