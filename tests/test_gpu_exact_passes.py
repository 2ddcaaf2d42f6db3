"""The FP64-exact passes of LPs too large to be launched early
(kernels_exact.cu: more than 8,192 warps), against the oracle bit for bit: rows
of one thread, of one warp loaded round by round, and of one warp with the next
rounds in flight (where the longest row is at least a 2,000th of all entries)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LPS = {
    "one_warp_fewer": lambda L: L.random_equality_lp(64, 32 * 8192 - 96, 2, seed=1),   # still early
    "short_rows": lambda L: L.random_equality_lp(300_000, 40_000, 4, seed=2),
    "warp_rows": lambda L: L.random_equality_lp(20_000, 270_000, 3, seed=3),
    "chains": lambda L: L.transportation_lp(300, 1000, seed=4),
    "a_long_chain": lambda L: L.badly_scaled_lp(20_000, 270_000, 4, seed=5),
}


@pytest.mark.parametrize("name", sorted(LPS))
@pytest.mark.parametrize("iters", [3, 45])
def test_passes_are_the_oracles(pkg, orc, name, iters):
    p = LPS[name](pkg.lpgen)
    o = orc.oracle_solve(p, max_iterations=iters)
    with pkg.Engine(0) as e:
        e.load(p)
        r = e.solve(pkg.PdhgOptions(max_iterations=iters))
    assert (r.status, r.iterations, r.restarts) == (o.status, o.iterations, o.restarts)
    assert r.operator_norm_estimate == o.operator_norm_estimate
    np.testing.assert_array_equal(r.primal, o.primal)
    np.testing.assert_array_equal(r.dual, o.dual)
    assert r.objective == o.objective
