"""Row blocks of the 2D column-march kernels: grids whose blocks are one row
(every warp of the GPU idle but for a few), a few rows with a short last
block, and more rows than resident warps, against the CPU oracle -- bit for
bit in the reference order, and to the contracted build's 1e-12 (two steps of
well under 200 rounded terms each: 2 * 200 * 2^-53 = 4.4e-14)."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import Solver
from helpers import rel_diff, same
from pyoracle import OracleGrid

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2), (28, 3), (29, 700), (61, 1777), (300, 131), (3, 2500)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("split", ["unsplit", "strang"])
@pytest.mark.parametrize("precision", ["fp64", "fp64_fma"])
def test_acoustics(shape, split, precision):
    bc = ("wall", "extrap", "periodic", "periodic")
    rd, solver, params, q0, _ = problems.random_acoustics_2d(*shape, seed=shape[1], bc=bc)
    rd.clawdata.dimensional_split = split
    _compare(rd, solver, params, q0, None, precision, 0.2 / max(shape))


# (three cells across the radius put ghost cells beyond the centre: no capacity there)
@pytest.mark.parametrize("shape", SHAPES[1:-1])
@pytest.mark.parametrize("precision", ["fp64", "fp64_fma"])
def test_annulus(shape, precision):
    rd, solver, params, q0, aux = problems.advection_2d_annulus(mx=shape[0], my=shape[1])
    _compare(rd, solver, params, q0, aux, precision, 0.1 / max(shape))


def _compare(rd, solver, params, q0, aux, precision, dt):
    g, o = Solver(rd.clawdata, solver, params, precision=precision), OracleGrid(rd.clawdata, solver, params)
    for s in (g, o):
        s.set_q(q0)
        if aux is not None:
            s.set_aux(aux)
    for _ in range(2):
        assert g.step(dt) == o.step(dt)
    q, r = g.get_q(), o.get_q()
    assert same(q, r) if precision == "fp64" else np.all(rel_diff(q, r) <= 1e-12)
    g.close()
