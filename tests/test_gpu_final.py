"""The result's sums: FP64-exact adds objective and dual objective in the
reference's order from staged rounds (kernels_exact.cu cta_ordered_sum), the
throughput modes over the row tiers with split rows (kernels_fast.cu
fast_final)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 1023, 1024, 1025, 2047, 2048, 2055])
@pytest.mark.parametrize("free", [-1, 0, 1000])  # a free column: the dual sum stops there
def test_exact_sums_are_the_oracles(pkg, orc, n, free):
    p = pkg.lpgen.random_equality_lp(max(1, n // 3), n, 1, seed=n)
    if 0 <= free < n:
        p.col_lo[free], p.col_hi[free] = -np.inf, np.inf
    with pkg.Engine(0) as e:
        e.load(p)
        r = e.solve(pkg.PdhgOptions(max_iterations=45))
    ref = orc.oracle_solve(p, max_iterations=45)
    assert r.objective == ref.objective
    assert r.duality_gap == ref.duality_gap
    np.testing.assert_array_equal(r.reduced_costs, ref.reduced_costs)


def test_fast_result_over_the_row_tiers(pkg):
    """Rows of A and columns (rows of A^T) in every tier, two of them split;
    each product of up to 9,000 terms of magnitude |a x| is within
    9,000 eps sum |a x| of numpy's."""
    rng = np.random.default_rng(3)
    wide = pkg.lpgen.row_lengths_lp([0, 1, 31, 32, 33, 511, 512, 513, 4096, 4097, 9000], 9001, seed=1)
    rows, cols = [], []
    for j, k in enumerate([1, 32, 33, 513, 4097, 9000]):  # long columns
        rows.append(np.sort(rng.choice(9001, size=k, replace=False)))
        cols.append(np.full(k, j))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    tall = pkg.Problem.from_coo(9001, 6, rows, cols, rng.standard_normal(rows.size), c=np.ones(6),
                                col_lo=np.zeros(6), col_hi=np.full(6, 5.0), row_lo=np.full(9001, -9.0),
                                row_hi=np.full(9001, 9.0))
    for p in (wide, tall):
        for precision in ("mixed", "fp64"):
            with pkg.Engine(0) as e:
                e.load(p)
                r = e.solve(pkg.PdhgOptions(max_iterations=50, precision=precision))
            row_of = np.repeat(np.arange(p.m), np.diff(p.row_ptr))
            aty = np.bincount(p.col_idx, weights=p.val * r.dual[row_of], minlength=p.n)
            mag = np.bincount(p.col_idx, weights=np.abs(p.val * r.dual[row_of]), minlength=p.n)
            eps = 9000 * np.finfo(float).eps
            assert np.all(np.abs(r.reduced_costs - (p.c - aty)) <= eps * (mag + np.abs(p.c)))
            act = np.bincount(row_of, weights=p.val * r.primal[p.col_idx], minlength=p.m)
            amag = np.bincount(row_of, weights=np.abs(p.val * r.primal[p.col_idx]), minlength=p.m)
            pinf = np.max(np.maximum(np.maximum(p.row_lo - act, act - p.row_hi), 0.0))
            assert abs(r.primal_infeasibility - pinf) <= eps * np.max(amag)
            assert abs(r.objective - p.c @ r.primal) <= eps * np.sum(np.abs(p.c * r.primal))
