"""The operator norm's estimate on both sides of the line up to which the power
iteration's launches start early (4,194,304 entries, engine.cu operator_norm):
the oracle's bit for bit in FP64-exact, within rounding where the rows are
summed over the tiers."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("supplies,demands", [(1000, 2097), (1024, 2048), (1100, 2500)])
def test_estimate(pkg, orc, supplies, demands):
    p = pkg.lpgen.transportation_lp(supplies, demands, seed=11)
    ref = orc.oracle_solve(p, max_iterations=1).operator_norm_estimate
    with pkg.Engine(0) as e:
        e.load(p)
        assert e.solve(pkg.PdhgOptions(max_iterations=1)).operator_norm_estimate == ref
        for precision in ("mixed", "fp64"):
            got = e.solve(pkg.PdhgOptions(max_iterations=1, precision=precision)).operator_norm_estimate
            assert abs(got - ref) <= 1e-12 * ref
