"""Each limiter's own kernels (and the run-time one for two different limiters,
none and Beam-Warming) against the CPU oracle on random data, where every
branch of phi is taken: bit for bit in the reference order; otherwise two steps
of well under 200 rounded terms, 2 * 200 * 2^-53 = 4.4e-14 (bar 1e-12) in FP64
and 2 * 200 * 2^-24 = 2.4e-5 (bar 5e-5) in FP32."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import rel_diff, same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu

LIMITERS = [["minmod"] * 2, ["superbee"] * 2, ["vanleer"] * 2, ["mc"] * 2, ["minmod", "superbee"],
            ["none", "none"], ["beamwarming"] * 2]
PRECISIONS = [("fp64", 0), ("fp64_fma", 1e-12), ("fp32", 5e-5)]


def _compare(rd, solver, params, q0, aux, precision, tol, dt):
    g, o = Solver(rd.clawdata, solver, params, precision=precision), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        if aux is not None:
            s.set_aux(aux)
    for _ in range(2):
        cg, co = g.step(dt), o.step(dt)
        assert cg == co if precision != "fp32" else abs(cg - co) <= 1e-6 * co
    q, r = g.get_q(), o.get_q()
    assert same(q, r) if tol == 0 else np.all(rel_diff(q, r) <= tol)
    g.close()


@pytest.mark.parametrize("limiter", LIMITERS)
@pytest.mark.parametrize("split", ["unsplit", "godunov", "strang"])
@pytest.mark.parametrize("precision,tol", PRECISIONS)
def test_plane(limiter, split, precision, tol):
    for shape, bc in (((61, 35), ("wall", "extrap", "periodic", "periodic")), ((125, 9), ("extrap",) * 4)):
        rd, solver, params, q0, _ = problems.random_acoustics_2d(*shape, seed=5, bc=bc)
        rd.clawdata.dimensional_split, rd.clawdata.limiter = split, list(limiter)
        _compare(rd, solver, params, q0, None, precision, tol, 0.2 / max(shape))


@pytest.mark.parametrize("limiter", LIMITERS)
@pytest.mark.parametrize("precision,tol", PRECISIONS)
def test_box(limiter, precision, tol):
    bc = ("periodic", "periodic", "wall", "extrap", "extrap", "wall")
    rd, solver, params, q0, aux = problems.random_acoustics_3d(30, 13, 9, seed=5, bc=bc)
    rd.clawdata.limiter = list(limiter)
    _compare(rd, solver, params, q0, aux, precision, tol, 0.004)


@pytest.mark.parametrize("limiter", LIMITERS)
@pytest.mark.parametrize("mx", [61, 600])
def test_line(limiter, mx):
    rd, solver, params, _, _ = problems.acoustics_1d_config(mx=mx)
    rd.clawdata.limiter = list(limiter)
    q0 = np.random.default_rng(mx).standard_normal((2, mx))
    _compare(rd, solver, params, q0, None, "fp64", 0, 0.3 / mx)
