"""FP32 media whose impedances leave FP32's range when multiplied (Z of 2^+-100).

Multiplying Z and the pressure by a power of two multiplies the step's
pressures by it and leaves the velocities alone, exactly, once 1 + Z Z' of the
limiter's products rounds to Z Z' (Z beyond 2^12) or to 1 (Z below 2^-12): so
the steps at 2^30 and 2^100, and at 2^-30 and 2^-100, are equal bit for bit
after scaling."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import rel_diff
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu


def _run(k, limiters, trans, bc):
    rd, solver, params, q0, aux = problems.random_acoustics_3d(37, 15, 11, seed=9, trans=trans, bc=bc)
    rd.clawdata.limiter = list(limiters)
    rd.clawdata.steps_max = 4
    q, a = np.float32(q0).astype(np.float64), np.float32(aux).astype(np.float64)
    q[0] *= 2.0**k
    a[0] *= 2.0**k
    s = Solver(rd, solver, params, "fp32")
    s.set_aux(a)
    s.set_q(q)
    info, st = s.advance(0.0, 1.0, 0.01)
    out = s.get_q()
    s.close()
    out[0] /= 2.0**k
    return out, (info, st["t_reached"], st["dt_next"])


@pytest.mark.parametrize("limiters,trans,bc", [
    (("mc", "mc"), 22, ("wall", "extrap", "periodic", "periodic", "extrap", "wall")),
    (("vanleer", "vanleer"), 22, ("extrap",) * 6),
    (("superbee", "minmod"), 11, ("periodic",) * 4 + ("wall",) * 2),
    (("minmod", "none"), 0, ("extrap",) * 6)])
@pytest.mark.parametrize("near,far", [(30, 100), (30, 62), (-30, -100), (-30, -62)])
def test_scaled_medium(near, far, limiters, trans, bc):
    (a, sa), (b, sb) = _run(near, limiters, trans, bc), _run(far, limiters, trans, bc)
    assert np.isfinite(a).all() and sa == sb
    assert np.array_equal(a, b)


@pytest.mark.parametrize("low,high", [(-45, 20), (45, -20), (-90, -60), (90, 20)])
def test_contrast(low, high):
    """Layers of very different Z, the first beyond the range in which the tile
    keeps the plain unit, against the oracle.  Two steps of under 200 rounded
    terms each of the size of the field: 2 * 200 * 2^-24 = 2.4e-5 (bar: 5e-5)."""
    rd, solver, params, q0, aux = problems.random_acoustics_3d(30, 12, 14, seed=3, limiter="mc")
    q, a = np.float32(q0).astype(np.float64), np.float32(aux).astype(np.float64)
    a[0, :9] *= 2.0**low
    a[0, 9:] *= 2.0**high
    g, o = Solver(rd.clawdata, solver, params, "fp32"), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q)
        s.set_aux(a)
    for dt in (0.004, 0.006):
        g.step(dt)
        o.step(dt)
    out = g.get_q()
    g.close()
    assert np.isfinite(out).all() and np.all(rel_diff(out, o.get_q()) <= 5e-5)
