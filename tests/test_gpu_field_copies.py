"""Host arrays in and out of the device fields: every route of the copy (the
dense staging buffer, a block above its size, unpadded rows, FP32) puts each element at its
place in the padded device rows and gives the same array back."""

import ctypes

import numpy as np
import pytest

from classic_b200 import problems
from classic_b200._lib import check

pytestmark = pytest.mark.gpu

STAGE = (8 << 20) // 8


def _device_rows(s, torch):
    ptr, es = ctypes.c_void_p(), ctypes.c_int()
    ld, fp = ctypes.c_longlong(), ctypes.c_longlong()
    check(s.lib.claw_q_device(s._h, ctypes.byref(ptr), ctypes.byref(es), ctypes.byref(ld), ctypes.byref(fp)),
          "claw_q_device")
    shape = s.q_shape
    rows = {2: [], 3: [ld.value], 4: [ld.value * shape[-2], ld.value]}[len(shape)]

    class V:
        __cuda_array_interface__ = {"shape": shape, "typestr": "<f%d" % es.value, "version": 3,
                                    "strides": tuple(es.value * x for x in [fp.value] + rows + [1]),
                                    "data": (ptr.value, False)}

    v = torch.as_tensor(V(), device="cuda").cpu().numpy()  # copied while s is alive
    assert s.q_shape == v.shape
    return v


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("cells", [(3, 2), (7, 5), (256, 3), (257, 131), (591, 591), (592, 592), (593, 593)])
def test_plane(cells, precision):
    import torch

    from classic_b200.solver import Solver

    assert (3 * cells[0] * cells[1] > STAGE) == (cells[0] >= 592)
    rd, name, params, _, _ = problems.radial_acoustics_2d(n=8)
    rd.clawdata.num_cells = list(cells)
    s = Solver(rd, name, params, precision=precision)
    q = np.random.default_rng(cells[0]).standard_normal(s.q_shape)
    want = q if precision == "fp64" else q.astype(np.float32)
    s.set_q(q)
    assert np.array_equal(_device_rows(s, torch), want)
    assert np.array_equal(s.get_q(), want)


@pytest.mark.parametrize("cells", [(5, 3, 2), (33, 300, 230)])
def test_box(cells):
    """More rows than a grid has blocks in y: 33 x 69,000."""
    import torch

    from classic_b200.solver import Solver

    rd, name, params, _, _ = problems.heterogeneous_acoustics_3d(n=4)
    rd.clawdata.num_cells = list(cells)
    for precision in ("fp64", "fp32"):
        s = Solver(rd, name, params, precision=precision)
        q = np.random.default_rng(1).standard_normal(s.q_shape).astype(np.float32).astype(np.float64)
        s.set_q(q)
        assert np.array_equal(_device_rows(s, torch), q)
        assert np.array_equal(s.get_q(), q)


def test_line():
    import torch

    from classic_b200.solver import Solver

    rd, name, params, _, _ = problems.acoustics_1d_config(mx=801)
    s = Solver(rd, name, params)
    q = np.random.default_rng(2).standard_normal(s.q_shape)
    s.set_q(q)
    assert np.array_equal(_device_rows(s, torch), q)
    assert np.array_equal(s.get_q(), q)


def test_batch():
    """One buffer for all instances: an instance above its size goes directly."""
    from classic_b200.solver import BatchSolver

    shapes = [(5, 9), (515, 515), (131, 64)]
    assert 4 * 515 * 515 > STAGE
    rds = [problems.euler_quadrants(shape=(4, 4))[0] for _ in shapes]
    for rd, shape in zip(rds, shapes):
        rd.clawdata.num_cells = list(shape)
    b = BatchSolver(rds, "euler_roe_2d", {"gamma": 1.4}, precision="fp64_fma")
    g = np.random.default_rng(3)
    qs = [g.standard_normal(b.q_shapes[k]) for k in range(len(shapes))]
    for k, q in enumerate(qs):
        b.set_q(k, q)
    for k, q in enumerate(qs):
        assert np.array_equal(b.get_q(k), q)
