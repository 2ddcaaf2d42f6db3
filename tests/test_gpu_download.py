"""A result's download (download.cuh): by the driver below 32 MB, by several
threads in pieces of 256 KB above, whose ends are ragged. Every entry is checked
against the others: one row per column with a column scaled by its number, so
the reduced cost of column j is c_j - a_j y_row and the row's activity a_j x_j.
Products of one entry: 4 eps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(16_384, 16_384), (2_000_000, 3), (2_097_152, 1), (2_097_153, 131_073), (1_700_001, 900_003)])
@pytest.mark.parametrize("batch", [False, True])
def test_every_entry_arrives(pkg, n, m, batch):
    j = np.arange(n)
    a = 1.0 + (j % 977) / 977.0
    p = pkg.Problem.from_coo(m, n, j % m, j, a, c=np.cos(j), col_lo=np.zeros(n), col_hi=np.full(n, 1.0 + j % 5),
                             row_lo=np.full(m, -1.0), row_hi=np.full(m, 0.5))
    opt = pkg.PdhgOptions(max_iterations=60, precision="fp64", tolerance=1e-12)
    with pkg.Engine(0) as e:
        if batch:
            small = pkg.lpgen.random_equality_lp(3, 5, 2, seed=1)
            e.load_batch([small, p])
            r = e.solve_batch(opt)[1]
        else:
            e.load(p)
            r = e.solve(opt)
    eps = 4 * np.finfo(float).eps
    assert np.any(r.dual != 0.0)
    assert np.all(np.abs(r.reduced_costs - (p.c - a * r.dual[j % m])) <= eps * (np.abs(p.c) + np.abs(a * r.dual[j % m])))
    assert np.all((r.primal >= 0.0) & (r.primal <= p.col_hi))
    assert abs(r.objective - p.c @ r.primal) <= 1e-11 * np.abs(p.c * r.primal).sum()
