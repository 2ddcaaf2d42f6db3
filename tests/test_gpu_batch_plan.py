"""Which batches run on clusters, and with how many CTAs an instance
(batch_resident.cuh plan_resident): told by a solve's launches (a power
iteration's four, one per class of clusters, or a graph and two per iteration
after the last check, and the result's two), and the points agree with the
single engine's either way (on the well-scaled LPs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IT = 83  # two check periods and a tail of three
POWER, OVER_ALL = 4 * 30, 1 + 2 * (IT % 40)


def eq(count, m, n, k):
    return lambda L: [L.random_equality_lp(m, n, k, seed=60 + i) for i in range(count)]


BATCHES = {  # precision, instances, launches beside the power iteration's and the result's
    "one_wave_of_sixteen": ("mixed", eq(7, 10000, 23000, 3), 1),
    "two_waves_of_sixteen": ("mixed", eq(16, 10000, 23000, 3), OVER_ALL),
    "wide_ones_among_many": ("mixed", lambda L: eq(8, 10000, 23000, 3)(L) + eq(120, 1000, 2500, 5)(L), 2),
    "sixteen_in_fp64": ("fp64", eq(16, 5000, 12500, 3), OVER_ALL),
    "as_many_as_run_at_once": ("fp64", eq(15, 300, 10000, 4), 1),
    "one_more": ("fp64", eq(16, 300, 10000, 4), 1),
    "a_long_row_in_fp64": ("fp64", lambda L: [L.badly_scaled_lp(4000, 9000, 6, seed=1)], OVER_ALL),
    "shorter_long_rows_in_fp64": ("fp64", lambda L: [L.badly_scaled_lp(500, 1200, 6, seed=i) for i in range(300)], 1),
    "a_long_row": ("mixed", lambda L: [L.badly_scaled_lp(4000, 9000, 6, seed=1)], 1),
}


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_route_and_points(pkg, name):
    precision, make, launches = BATCHES[name]
    ps = make(pkg.lpgen)
    opt = pkg.PdhgOptions(precision=precision, max_iterations=IT, tolerance=1e-30, autotune=False,
                          restart_rule="adaptive")
    with pkg.Engine(0) as e:
        e.load_batch(ps)
        rs = e.solve_batch(opt)
        assert rs[0].kernel_launches == POWER + launches + 2
        # nonexpansive iterations: IT x (terms of the longest row) x eps x the
        # points' magnitude apart, in FP32 64 eps for independent roundings; the
        # step sizes follow operator norms that agree to 1e-12
        for p, r in list(zip(ps, rs))[::7] if "long_row" not in name else []:
            e.load(p)
            s = e.solve(opt)
            assert r.status == s.status and r.iterations == s.iterations == IT and r.restarts == s.restarts
            eps = np.finfo(np.float32 if precision == "mixed" else np.float64).eps
            tol = IT * ((64 if precision == "mixed" else 1500) * eps + 1e-12)
            for u, v in ((r.primal, s.primal), (r.dual, s.dual)):
                assert np.max(np.abs(u - v)) <= tol * max(1.0, np.max(np.abs(v)))
