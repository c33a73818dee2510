"""Quotients by the capacity of a mapped 2D grid, formed from one reciprocal a
cell: bit for bit the CPU oracle's divisions, also where capacities or
numerators are too far from one for the correction steps and the division
itself takes over (2^+-100 and 2^+-896), on grids of one and several strips."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(28, 3), (61, 35)])
@pytest.mark.parametrize("cap_exp", [0, 99, 101, -99, -101])
@pytest.mark.parametrize("q_exp", [0, -940, 900])
@pytest.mark.parametrize("limiter", ["vanleer", "mc"])
def test_quotients(shape, cap_exp, q_exp, limiter):
    rd, solver, params, q0, aux = problems.advection_2d_annulus(mx=shape[0], my=shape[1])
    rd.clawdata.limiter = [limiter]
    aux = aux.copy()
    aux[rd.clawdata.capa_index - 1] *= 2.0 ** cap_exp  # a step 2^cap_exp as long does the same
    q0 = q0 * 2.0 ** q_exp
    g, o = Solver(rd.clawdata, solver, params, precision="fp64"), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        s.set_aux(aux)
    for _ in range(2):
        dt = 0.1 / max(shape) * 2.0 ** cap_exp
        assert g.step(dt) == o.step(dt)
        assert same(g.get_q(), o.get_q())
