"""A grid holds a staging buffer for its host copies only where a copy takes it:
not for a block of one field, an unpadded grid or a 1D one."""
import math

import pytest

from classic_b200 import problems
from classic_b200.solver import Solver

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _round(x, k):
    return (x + k - 1) // k * k


def _one_field():  # q 7.9 MiB, aux above the buffer's size
    return problems.advection_2d_annulus(mx=1000, my=1036)


def _unpadded():  # three fields of 512^2: 6 MiB
    return problems.random_acoustics_2d(512, 512)


def _line():  # two fields of 500,000: 7.6 MiB
    return problems.acoustics_1d_config(mx=500000)


@pytest.mark.parametrize("build", [_one_field, _unpadded, _line])
def test_no_buffer(build):
    import torch

    rd, solver, params, q0, aux = build()

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    Solver(rd, solver, params).close()  # what the first grid of a process loads
    before = used()
    s = Solver(rd, solver, params)
    held = used() - before
    row = q0.shape[-1] if q0.ndim == 2 else _round(q0.shape[-1], 32)
    fields = 2 * [8 * row * math.prod(q0.shape[:-1])]
    if aux is not None:
        fields.append(8 * _round(aux.shape[-1], 4) * math.prod(aux.shape[:-1]))
    # device memory comes in 2 MiB pages; the small blocks share one
    want = sum(_round(f, 2 * MIB) for f in fields) + 2 * MIB
    assert held <= want, (held / MIB, want / MIB)
    s.set_q(q0)
    assert (s.get_q() == q0).all()
    s.close()
