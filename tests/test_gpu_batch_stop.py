"""A stop request to a batch of more instances than run on the GPU at once
(batch_resident.cuh: an instance waits for a cluster's place): an instance that
runs ends after its check period, one that still waits ends without an
iteration, and each reports the iterations that its point has.

A wave of instances takes about 1.5 seconds here (hundreds of thousands of
iterations of 1 to 3 us), the time limit a part of that, and there are
three waves.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNT = 1700     # at most four of these instances to an SM
ITERS = 800_000


@pytest.fixture(scope="module")
def engine(pkg):
    with pkg.Engine(0) as e:
        e.load_batch([pkg.lpgen.random_equality_lp(60, 150, 5, seed=400 + i) for i in range(COUNT)])
        e.solve_batch(pkg.PdhgOptions(precision="mixed", max_iterations=40))  # kernels and buffers are there
        yield e


def stopped(pkg, engine, period, iters):
    rs = engine.solve_batch(pkg.PdhgOptions(precision="mixed", tolerance=1e-30, max_iterations=iters,
                                            restart_check_period=period, time_limit_seconds=0.6))
    ran = [r for r in rs if r.iterations > 0]
    waited = [r for r in rs if r.iterations == 0]
    assert ran and waited, (len(ran), len(waited))
    assert all(r.status == "time_limit" and not np.any(r.dual) for r in waited)
    assert all(np.any(r.dual) for r in ran)
    return ran


def test_a_running_instance_ends_after_its_period(pkg, engine):
    ran = stopped(pkg, engine, ITERS, 3 * ITERS)
    assert all(r.status == "time_limit" and r.iterations == ITERS for r in ran)


def test_an_instance_past_its_last_check_ends_its_iterations(pkg, engine):
    ran = stopped(pkg, engine, 2 * ITERS, ITERS)
    assert all(r.status == "iteration_limit" and r.iterations == ITERS for r in ran)
