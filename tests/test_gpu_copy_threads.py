"""Host copies of one object from several host threads (ctypes lets go of the
interpreter lock): instances of a batch, q and aux of one grid, share the
staging buffer of the object and must not see each other's data."""
import threading

import numpy as np
import pytest

from classic_b200 import problems
from classic_b200.solver import BatchSolver, Solver

pytestmark = pytest.mark.gpu


def _together(jobs):
    """Run the jobs on a thread each, started together; raise what they raise."""
    errors, start = [], threading.Barrier(len(jobs))

    def body(job):
        try:
            start.wait()
            job()
        except BaseException as e:  # noqa: BLE001 (handed to the caller)
            errors.append(e)

    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_batch_instances():
    """Padded instances above the 64 KB that go in directly, one thread each:
    values of their own in and out, again and again."""
    sizes = [(50, 49), (131, 64), (77, 90), (201, 150), (50, 49), (333, 97)]
    rds = [problems.euler_quadrants(shape=s)[0] for s in sizes]
    b = BatchSolver(rds, "euler_roe_2d", {"gamma": 1.4})

    def job(k):
        rng = np.random.default_rng(k)
        for _ in range(40):
            q = rng.standard_normal(b.q_shapes[k])
            b.set_q(k, q)
            for _ in range(3):
                assert np.array_equal(b.get_q(k), q), k

    _together([lambda k=k: job(k) for k in range(len(sizes))])
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_q_beside_aux(precision):
    rd, solver, params, q0, aux = problems.heterogeneous_acoustics_3d(shape=(33, 30, 29))
    s = Solver(rd, solver, params, precision)

    def fields():
        rng = np.random.default_rng(0)
        for _ in range(60):
            q = rng.standard_normal(q0.shape).astype(np.float32).astype(np.float64)
            s.set_q(q)
            assert np.array_equal(s.get_q(), q)

    def medium():
        for _ in range(120):
            s.set_aux(aux)

    _together([fields, medium])
    # the medium is whole too: a step equals that of a grid set up by one thread
    s.set_q(q0)
    s.step(1e-3)
    other = Solver(rd, solver, params, precision)
    other.set_aux(aux)
    other.set_q(q0)
    other.step(1e-3)
    assert np.array_equal(s.get_q(), other.get_q())
    s.close()
    other.close()
