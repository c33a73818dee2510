"""The 1D kernel's strips of 28 cells, bit for bit against the CPU oracle where
they can go wrong: one cell either side of a strip, of the 15 and 31 strips
that fill a CTA of 512 and 1024 threads (more strips than warps beyond), grids
too large for shared memory, the compiled and the run-time method, a rejected
first step and a source that needs dt before the waves."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu


def _compare(rd, solver, params, q0, aux, tend, dt, **kw):
    g, o = Solver(rd.clawdata, solver, params, **kw), OracleGrid(rd.clawdata, solver, params, **kw)
    for s in (g, o):
        s.set_q(q0)
        if aux is not None:
            s.set_aux(aux)
    (ig, sg), (io, so) = g.advance(0.0, tend, dt), o.advance(0.0, tend, dt)
    assert ig == io
    for key in ("t_reached", "dt_next", "steps_taken", "cfl_max_seen", "cfl_last", "dt_min"):
        assert sg[key] == so[key], key
    assert same(g.get_q(), o.get_q())
    g.close()


@pytest.mark.parametrize("mx", [2, 3, 27, 28, 29, 56, 419, 420, 421, 448, 867, 868, 869, 2500])
@pytest.mark.parametrize("lim", ["mc", "superbee"])
def test_acoustics(mx, lim):
    rd, solver, params, q0, aux = problems.acoustics_1d_config(mx=mx)
    rd.clawdata.limiter = [lim, lim]
    rd.clawdata.bc_lower[0], rd.clawdata.bc_upper[0] = "extrap", "wall"
    _compare(rd, solver, params, q0, aux, 12.0 / mx, 3.0 / mx)  # dt rejected once


@pytest.mark.parametrize("mx", [30, 421, 3000])
def test_heterogeneous_and_euler(mx):
    _compare(*problems.acoustics_1d_heterogeneous(mx=mx), tend=40.0 / mx, dt=20.0 / mx)
    _compare(*problems.euler_1d_wcblast(mx=mx), tend=0.3 / mx, dt=1e-6)


@pytest.mark.parametrize("mx", [12000, 30000])
def test_beyond_shared_memory(mx):
    rd, solver, params, q0, aux = problems.acoustics_1d_config(mx=mx)
    for lim in ("mc", "vanleer"):
        rd.clawdata.limiter = [lim, lim]
        _compare(rd, solver, params, q0, aux, 6.0 / mx, 3.0 / mx)


@pytest.mark.parametrize("mx", [40, 900])
@pytest.mark.parametrize("split", ["godunov", "strang"])
def test_radial_source(mx, split):
    rd, solver, params, q0, aux = problems.radial_acoustics_1d(mx=mx, order=2, source_split=split)
    _compare(rd, solver, params, q0, aux, 10.0 / mx, 4.0 / mx, user_source="radial")
