"""The power iteration's norm kernel against the oracle's recursion: the
estimate is the reference's bit for bit at every shape of the pairwise tree
(leaves, one CTA's subtree, several CTAs), and within rounding where the rows
are summed over the tiers."""
import pytest

pytestmark = pytest.mark.gpu

# n: one leaf, two leaves, a subtree's edges (32 nodes of up to 256), several CTAs
SIZES = [1, 2, 127, 128, 129, 255, 256, 257, 4096, 4097, 8191, 8192, 8193, 16385, 70001]


@pytest.mark.parametrize("n", SIZES)
def test_estimate_over_the_tree_shapes(pkg, orc, n):
    m = max(1, n // 3)
    p = pkg.lpgen.random_equality_lp(m, n, min(3, m), seed=n)
    ref = orc.oracle_solve(p, max_iterations=1).operator_norm_estimate
    with pkg.Engine(0) as e:
        e.load(p)
        assert e.solve(pkg.PdhgOptions(max_iterations=1)).operator_norm_estimate == ref
        fast = e.solve(pkg.PdhgOptions(max_iterations=1, precision="fp64")).operator_norm_estimate
    assert abs(fast - ref) <= 1e-12 * ref


@pytest.mark.parametrize("lengths,n", [([5] * 50 + [40, 600, 4097, 9000], 9001), ([0, 1, 33] * 7, 64)])
def test_estimate_over_the_row_tiers(pkg, orc, lengths, n):
    p = pkg.lpgen.row_lengths_lp(lengths, n, seed=5)
    ref = orc.oracle_solve(p, max_iterations=1).operator_norm_estimate
    with pkg.Engine(0) as e:
        e.load(p)
        assert e.solve(pkg.PdhgOptions(max_iterations=1)).operator_norm_estimate == ref
        for precision in ("mixed", "fp64"):
            got = e.solve(pkg.PdhgOptions(max_iterations=1, precision=precision)).operator_norm_estimate
            assert abs(got - ref) <= 1e-12 * ref
