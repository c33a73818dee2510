"""A batch beside other work on the GPU: its CTAs then start when the other
work's blocks make room, some after the first instances of the batch have
ended, and all must still agree on which rows are whose."""
import threading

import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import BatchSolver

pytestmark = pytest.mark.gpu

SIZES = [24, 30, 41, 56, 24, 75, 200, 33, 320, 28]  # the small ones end first


def _batch(seed):
    ins = [problems.euler_quadrants(n=n, seed=seed + k) for k, n in enumerate(SIZES)]
    b = BatchSolver([i[0] for i in ins], "euler_roe_2d", {"gamma": 1.4})
    return b, ins


def _run(b, ins):
    for k, i in enumerate(ins):
        b.set_q(k, i[3])
    info, st = b.advance(0.0, 0.1)
    for s in st:
        s.pop("device_ms"), s.pop("launches")
    return info, st, [b.get_q(k) for k in range(len(ins))]


def _equal(x, y):
    return x[:2] == y[:2] and all(np.array_equal(p, q, equal_nan=True) for p, q in zip(x[2], y[2]))


def test_beside_matmuls():
    import torch

    b, ins = _batch(900)
    alone = _run(b, ins)
    m = torch.randn(8192, 8192, device="cuda", dtype=torch.bfloat16)
    out = torch.empty_like(m)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(4):
        with torch.cuda.stream(side):
            for _ in range(60):  # about 45 ms of the whole GPU
                torch.matmul(m, m, out=out)
        assert _equal(_run(b, ins), alone)
        torch.cuda.synchronize()
    b.close()


def test_two_batches():
    pairs = [_batch(900), _batch(950)]
    alone = [_run(*p) for p in pairs]
    good = [0, 0]

    def body(k):
        for _ in range(8):
            good[k] += _equal(_run(*pairs[k]), alone[k])

    threads = [threading.Thread(target=body, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert good == [8, 8]
    for p in pairs:
        p[0].close()
