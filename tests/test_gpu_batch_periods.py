"""A batch on clusters (batch_resident.cuh) over several check periods, against
the kernels over all instances, which a batch takes when one of its instances
fits no cluster: sums carried over a period that ends without a restart, FP32
sums folded into them, restarts to an average over two periods, the primal
weight's later updates; in FP64 on every class of clusters.

Six periods and a tail: the adaptive rule restarts at the latest when a span is
36% of all iterations, so the third check passes without one and the fourth
restarts to the average of two periods. The launches of a solve tell the paths
apart (test_gpu_batch_tail.py).

Tolerances: a PDHG iteration is nonexpansive and an average no larger than its
points, so after `IT` iterations the paths differ by at most IT x (terms of the
longest row, 1,500) x eps x the points' magnitude; FP32: 64 eps for independent
roundings. With the primal weight, whose step sizes take over the points'
relative difference, every iteration may add that difference again: IT times
as much, which leaves nothing to compare in FP32.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IT = 247
POWER = 4 * 30
SIZES = {"fp64": [(60, 150, 5), (220, 520, 6), (600, 1000, 3), (500, 1200, 5), (2000, 3000, 4), (3000, 9000, 7),
                  (2000, 9000, 16), (5000, 12500, 3)],
         "mixed": [(60, 150, 5), (500, 1200, 5), (2000, 5000, 7), (3000, 9000, 7), (5000, 15000, 7)]}
CLASSES = {"fp64": 7, "mixed": 5}  # of clusters, at most


@pytest.mark.parametrize("precision,halpern,weight", [("fp64", False, False), ("fp64", False, True),
                                                      ("fp64", True, True), ("mixed", False, False),
                                                      ("mixed", True, False)])
@pytest.mark.parametrize("copies", [1, 20])  # clusters for each instance's time; for the SMs'
def test_periods_reach_the_points_of_the_kernels_over_all(pkg, precision, halpern, weight, copies):
    L = pkg.lpgen
    ps = [L.random_equality_lp(*size, seed=900 * i + j) for i in range(copies) for j, size in enumerate(SIZES[precision])]
    ps.append(L.row_lengths_lp([0, 1, 31, 32, 33, 511, 512, 513, 0, 1100, 1500], 1501, seed=3))
    rules = dict(termination_rule="relative_kkt_l2", restart_rule="adaptive_l2") if halpern else dict(
        restart_rule="adaptive")
    opt = pkg.PdhgOptions(max_iterations=IT, tolerance=1e-30, precision=precision, halpern=halpern, autotune=False,
                          primal_weight_update=weight, **rules)
    got = []
    for batch in (ps, ps + [L.random_equality_lp(20000, 60000, 3, seed=9)]):
        with pkg.Engine(0) as e:
            e.load_batch(batch)
            got.append(e.solve_batch(opt))
    tail = 2 * (IT % 40)
    assert POWER + 2 < got[0][0].kernel_launches <= POWER + CLASSES[precision] + 2
    assert got[1][0].kernel_launches == POWER + 1 + tail + 2
    eps = np.finfo(np.float32 if precision == "mixed" else np.float64).eps
    tol = IT * (64 if precision == "mixed" else 1500) * eps * (IT if weight else 1)
    assert any(3 <= a.restarts < 6 for a in got[0])  # some checks without a restart before one with
    for p, a, b in zip(ps, *got):
        assert a.status == b.status == "iteration_limit" and a.iterations == b.iterations == IT
        for u, v in ((a.primal, b.primal), (a.dual, b.dual)):
            assert np.max(np.abs(u - v), initial=0.0) <= tol * max(1.0, np.max(np.abs(v), initial=0.0)), (p.m, p.n)


def test_a_stalled_instance_goes_on_in_fp64_off_the_clusters(pkg):
    # 5,000 x 15,000 fits a cluster in FP32 only: the FP64 phase runs on the
    # kernels over all instances (a graph; three classes of clusters before)
    ps = [pkg.lpgen.random_equality_lp(*size, seed=50 + i) for i, size in enumerate(
        [(60, 150, 5), (500, 1200, 5), (5000, 15000, 7)])]
    opt = dict(tolerance=1e-8, max_iterations=400_000, termination_rule="relative_kkt", restart_rule="adaptive",
               primal_weight_update=True)
    with pkg.Engine(0) as e:
        e.load_batch(ps)
        rs = e.solve_batch(pkg.PdhgOptions(precision="mixed", **opt))
        assert rs[0].kernel_launches == POWER + 3 + 1 + 1 + 4  # the clusters, the widening, the graph, the results
    for p, r in zip(ps, rs):
        assert r.status == "optimal" and 0 < r.fp64_iterations < r.iterations
        # the rule's three parts, restated (equality rows, boxed columns)
        row = np.repeat(np.arange(p.m), np.diff(p.row_ptr))
        act = np.bincount(row, p.val * r.primal[p.col_idx], p.m)
        rc = p.c - np.bincount(p.col_idx, p.val * r.dual[row], p.n)
        dual = p.row_lo @ r.dual + np.sum(np.where(rc > 0, rc * p.col_lo, rc * p.col_hi))
        obj = p.c @ r.primal
        assert np.max(np.abs(act - p.row_lo)) <= 2e-8 * (1.0 + np.max(np.abs(p.row_lo)))
        assert np.max(np.abs(rc - r.reduced_costs)) <= 1e-9 * max(1.0, np.max(np.abs(rc)))
        assert abs(obj - dual) <= 2e-8 * (1.0 + abs(obj) + abs(dual))
