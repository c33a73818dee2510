"""The contracted / FP32 3D step (step3f_kernel) against the CPU oracle where
its tiles can go wrong: one cell either side of the 28-column tiles, of the
10-row (FP64) and 7-row (FP32) tiles and of the two-cell minimum, every kind
of boundary, and the piston at z-upper.

Tolerances: a step adds well under 200 rounded terms of the size of q to a
cell, so two steps stay within 2 * 200 * 2^-24 = 2.4e-5 in FP32 (bar: 5e-5);
in FP64 the same count gives 4.4e-14 (bar: 1e-12, the contracted build's)."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import rel_diff
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu

SHAPES = [(27, 9, 5), (28, 10, 6), (29, 11, 7), (30, 6, 33), (56, 20, 4), (57, 21, 3), (26, 7, 2),
          (3, 8, 40), (58, 14, 9), (2, 15, 2)]
BCS = [("periodic", "periodic", "wall", "extrap", "extrap", "wall"),
       ("wall", "extrap", "periodic", "periodic", "periodic", "periodic")]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bc", BCS)
@pytest.mark.parametrize("precision,tol", [("fp64_fma", 1e-12), ("fp32", 5e-5)])
def test_tile_edges(shape, bc, precision, tol):
    rd, solver, params, q0, aux = problems.random_acoustics_3d(*shape, seed=sum(shape), bc=bc)
    g, o = Solver(rd.clawdata, solver, params, precision=precision), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        s.set_aux(aux)
    t = 0.0
    for dt in (0.004, 0.006):
        cg, co = g.step(dt), o.step(dt, t)
        t += dt
        assert cg == co if precision == "fp64_fma" else abs(cg - co) <= 1e-6 * co
    assert np.all(rel_diff(g.get_q(), o.get_q()) <= tol)
    g.close()


@pytest.mark.parametrize("precision,tol", [("fp64_fma", 1e-12), ("fp32", 5e-5)])
def test_piston(precision, tol):
    rd, solver, params, q0, aux = problems.acoustics_3d_heterogeneous(n=20)
    g = Solver(rd.clawdata, solver, params, precision=precision, user_bc="piston")
    o = OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        s.set_aux(aux)
    t = 0.0
    for _ in range(4):
        g.step(0.02)
        o.step(0.02, t)
        t += 0.02
    q, r = g.get_q(), o.get_q()
    assert np.abs(r[0]).max() > 1e-3
    assert np.max(np.abs(q - r)) <= tol * np.abs(r).max()
    g.close()
