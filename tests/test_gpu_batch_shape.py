"""The batch's launch shape: what the autotuner returns is what it keeps, so
that setting it again changes nothing, and every tile height gives the same
bits in the reference's order of operations (the contracted build rounds a
tile's first row differently, as it always has)."""
import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import BatchSolver

pytestmark = pytest.mark.gpu

SIZES = [60, 130, 200]


def _batch(precision):
    ins = [problems.euler_quadrants(n=n, seed=40 + k) for k, n in enumerate(SIZES)]
    return BatchSolver([i[0] for i in ins], "euler_roe_2d", {"gamma": 1.4}, precision), ins


def _advance(b, ins):
    for k, i in enumerate(ins):
        b.set_q(k, i[3])
    info, stats = b.advance(0.0, 0.05)
    assert info == 0
    return stats[0]["device_ms"], [b.get_q(k) for k in range(len(ins))]


def test_returned_shape_is_the_kept_one():
    """These grids' steps take two to eight times as long in tiles of 16 rows and
    more as in shares of one, so a time within 1.5 of the tuned one tells."""
    b, ins = _batch("fp64_fma")
    for k, i in enumerate(ins):
        b.set_q(k, i[3])
    shape = b.autotune(repeats=3)
    tuned = min(_advance(b, ins)[0] for _ in range(5))
    b.set_shape(shape["min_rows"], shape["ctas_per_sm"])
    again = min(_advance(b, ins)[0] for _ in range(5))
    b.close()
    assert max(tuned, again) <= 1.5 * min(tuned, again), (shape, tuned, again)


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 48, 1000])
def test_heights_agree(rows):
    b, ins = _batch("fp64")
    base = _advance(b, ins)[1]
    b.set_shape(rows, 2)
    other = _advance(b, ins)[1]
    b.close()
    assert all(np.array_equal(x, y) for x, y in zip(base, other))
