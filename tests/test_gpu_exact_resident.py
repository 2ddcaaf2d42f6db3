"""FP64-exact iterations of a small LP in one launch of one cluster
(exact_resident.cu) against the passes: a traced solve runs those, iterate by
iterate, and both keep the reference's order, so the two end in the same bits.
Sizes: one row, one CTA of 256 and of 1,024 threads, clusters, empty rows, rows
up to and past the longest it takes; whole periods and a cut one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LPS = {
    "one_row": (lambda L: L.random_equality_lp(1, 2, 1, seed=1), True),
    "few_threads": (lambda L: L.random_equality_lp(60, 150, 5, seed=2), True),
    "edge_of_a_slice": (lambda L: L.random_equality_lp(33, 65, 3, seed=3), True),
    "one_cta": (lambda L: L.random_equality_lp(350, 801, 5, seed=4), True),
    "two": (lambda L: L.random_equality_lp(700, 1503, 6, seed=5), True),
    "eight": (lambda L: L.random_equality_lp(2000, 5000, 7, seed=6), True),
    "sixteen": (lambda L: L.random_equality_lp(2800, 7001, 9, seed=7), True),
    "past_sixteen": (lambda L: L.random_equality_lp(3000, 9001, 9, seed=7), False),
    "rows_of_128": (lambda L: L.row_lengths_lp([0, 1, 31, 32, 33, 0, 127, 128] * 3, 200, seed=8), True),
    "row_of_129": (lambda L: L.row_lengths_lp([0, 1, 31, 32, 33, 0, 127, 129] * 3, 200, seed=8), False),
    "too_large": (lambda L: L.random_equality_lp(9000, 17000, 4, seed=9), False),
}


@pytest.mark.parametrize("name", sorted(LPS))
@pytest.mark.parametrize("iters", [1, 40, 173])
def test_a_period_in_one_launch_is_its_passes(pkg, name, iters):
    make, resident = LPS[name]
    with pkg.Engine(0) as e:
        e.load(make(pkg.lpgen))
        a = e.solve(pkg.PdhgOptions(max_iterations=iters))
        b = e.solve(pkg.PdhgOptions(max_iterations=iters, trace_iters=iters))
    assert (a.kernel_launches < b.kernel_launches) == resident
    assert (a.status, a.iterations, a.restarts) == (b.status, b.iterations, b.restarts)
    for f in ("primal", "dual", "reduced_costs"):
        np.testing.assert_array_equal(getattr(a, f), getattr(b, f))
    assert a.objective == b.objective and a.relative_kkt == b.relative_kkt
