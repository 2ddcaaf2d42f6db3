"""Columns of two entries given by runs (intake.cu k_col_runs) on the wide
primal pass (kernels_fast.cu fast_primal_wide) and in the check, against the
passes that load every column index: the same arithmetic, so the same bits.
(The points' bits: the check's sums over the LP take a split row's terms in the
CTA that completes the row, so their last bits vary from run to run.)
Sizes: fewer columns than a vector or a run, remainders of both, runs broken by
a row's end and by shuffled columns, launched early and not (4M entries)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lp(pkg, m, n, boxed, shuffled):
    rng = np.random.default_rng(m * n)
    cols = m * n
    i, j = np.divmod(np.arange(cols), n)
    if shuffled:  # the last eighth in another order: its descriptors are no runs
        k = cols - cols // 8
        p = np.concatenate([np.arange(k), k + rng.permutation(cols - k)])
        i, j = i[p], j[p]
    hi = rng.uniform(0.5, 2.0, cols) if boxed else np.full(cols, 2.0)
    c = np.arange(cols)
    return pkg.Problem.from_coo(m + n, cols, np.concatenate([i, m + j]), np.concatenate([c, c]),
                                rng.uniform(0.5, 1.5, 2 * cols), c=rng.standard_normal(cols), col_lo=np.zeros(cols),
                                col_hi=hi, row_lo=np.full(m + n, -np.inf), row_hi=rng.uniform(0.5, 1.0, m + n))


@pytest.mark.parametrize("m,n", [(1, 1), (1, 3), (3, 5), (1, 33), (7, 31), (5, 64), (40, 67), (1100, 2001)])
@pytest.mark.parametrize("boxed,shuffled", [(False, False), (True, False), (True, True)])
def test_runs_give_the_loaded_columns_bits(pkg, monkeypatch, m, n, boxed, shuffled):
    p = lp(pkg, m, n, boxed, shuffled)
    rules = dict(termination_rule="relative_kkt_l2", restart_rule="adaptive_l2")
    for precision in ("mixed", "fp64"):
        for form in (dict(), dict(halpern=True, **rules)):
            opt = pkg.PdhgOptions(max_iterations=95, tolerance=1e-12, precision=precision, autotune=False, **form)
            got = []
            for knob in ("1", "0"):  # "0": every column index is loaded
                monkeypatch.setenv("PDHG_B200_DENSE_ROWS", knob)
                with pkg.Engine(0) as e:
                    e.load(p)
                    got.append(e.solve(opt))
            np.testing.assert_array_equal(got[0].primal, got[1].primal)
            np.testing.assert_array_equal(got[0].dual, got[1].dual)
            assert got[0].restarts == got[1].restarts
