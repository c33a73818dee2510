"""The reference-order 3D sweeps' quotients bit for bit against the CPU oracle
where their quick form ends: fluctuations at and below its smallest size
(2^-896, about 1e-270) down to subnormals, zero next to them, impedance sums
beyond 2^100 and media across it within one tile, and values near its largest."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("amplitude", [1e-320, 1e-300, 1e-270, 1e-140, 1e140, 1e260])
@pytest.mark.parametrize("impedance", [1.0, 1e31, 1e-33])
def test_extremes(amplitude, impedance):
    rd, solver, params, q0, aux = problems.random_acoustics_3d(19, 13, 11, seed=4)
    rng = np.random.default_rng(5)
    q0 = q0 * amplitude
    q0[:, :, :, :6] = 0.0
    q0[0] *= np.where(rng.uniform(size=q0[0].shape) < 0.2, 1e-40, 1.0)
    aux[0] *= np.where(np.arange(aux.shape[3]) < 12, 1.0, impedance)
    g, o = Solver(rd.clawdata, solver, params), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        s.set_aux(aux)
    for k in range(2):
        with np.errstate(all="ignore"):
            assert g.step(0.01) == o.step(0.01, 0.01 * k)
    assert same(g.get_q(), o.get_q())
    g.close()
