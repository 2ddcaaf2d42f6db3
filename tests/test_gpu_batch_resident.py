"""A batch whose instances run on one cluster each (batch_resident.cu) against
the kernels over all instances (batch_kernels.cu), which a batch takes when one
of its instances fits no cluster: the same batch with such an instance added.

A row's products are summed in another order (other lanes per row). A PDHG
iteration is nonexpansive, so after `it` iterations the paths differ by at most
it x (terms of the longest row, 1,500) x eps x the points' magnitude; in FP32,
where that is loose, by the 64 eps that 1,500 independent roundings give.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IT = 47  # a whole check period and a tail


def lps(pkg, seed):
    """Sizes around each class of CTAs (256, 512 and 1,024 threads, clusters,
    entries in global memory), and rows of A and of A^T in every tier."""
    gen = pkg.lpgen
    out = [gen.random_equality_lp(m, n, k, seed=seed + i) for i, (m, n, k) in enumerate(
        [(1, 1, 1), (1, 7, 1), (3, 5, 2), (60, 150, 5), (600, 1000, 3), (500, 1200, 5), (2000, 3000, 4),
         (2000, 5000, 7), (3000, 9000, 7), (5000, 15000, 7), (2000, 9000, 16)])]
    out.append(gen.row_lengths_lp([0, 1, 31, 32, 33, 511, 512, 513, 0, 1100, 1500], 1501, seed=seed))
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for j, k in enumerate([0, 1, 32, 511, 512, 513, 1100]):  # the same lengths as columns
        rows.append(np.sort(rng.choice(1101, size=k, replace=False)))
        cols.append(np.full(k, j))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    out.append(pkg.Problem.from_coo(1101, 7, rows, cols, rng.standard_normal(rows.size), c=np.ones(7),
                                    col_lo=np.zeros(7), col_hi=np.full(7, 5.0), row_lo=np.full(1101, -9.0),
                                    row_hi=np.full(1101, 9.0)))
    return out


@pytest.mark.parametrize("halpern", [False, True])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("copies", [1, 20])  # clusters for each instance's time; for the SMs'
def test_clusters_reach_the_points_of_the_kernels_over_all(pkg, halpern, precision, copies):
    batch = [p for i in range(copies) for p in lps(pkg, 100 * i)]
    large = pkg.lpgen.random_equality_lp(20000, 60000, 3, seed=9)
    rules = dict(termination_rule="relative_kkt_l2", restart_rule="adaptive_l2") if halpern else dict(
        restart_rule="adaptive")
    opt = pkg.PdhgOptions(max_iterations=IT, tolerance=1e-12, precision=precision, halpern=halpern, autotune=False,
                          primal_weight_update=True, **rules)
    got = []
    for ps in (batch, batch + [large]):
        with pkg.Engine(0) as e:
            e.load_batch(ps)
            got.append(e.solve_batch(opt))
    eps = np.finfo(np.float32 if precision == "mixed" else np.float64).eps
    for p, a, b in zip(batch, *got):
        assert a.status == b.status and a.iterations == b.iterations
        tol = IT * 1500 * eps if precision == "fp64" else IT * 64 * eps
        for u, v in ((a.primal, b.primal), (a.dual, b.dual)):
            scale = max(1.0, np.max(np.abs(v), initial=0.0))
            assert np.max(np.abs(u - v), initial=0.0) <= tol * scale, (p.m, p.n)
