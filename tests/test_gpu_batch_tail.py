"""A batch on clusters with fewer iterations than a check period: no period and
no check, only the tail (batch_resident.cuh), against the kernels over all
instances, which a batch takes when one of its instances fits no cluster.

Sizes: an instance on a cluster of two CTAs, of eight and of sixteen (the last
two with their entries in global memory). The launches of a solve tell the
paths apart: a power iteration's four, one per class of clusters or two per
iteration, the result's two. Tolerances: a PDHG iteration is nonexpansive, so
after `it` iterations the paths differ by at most it x (terms of the longest
row, below 1,500) x eps x the points' magnitude; FP32: 64 eps for independent
roundings.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = {"mixed": [(1900, 2700, 3), (5000, 15000, 7), (10000, 23000, 3)],
         "fp64": [(700, 1700, 5), (3000, 9000, 7), (5000, 12500, 3)]}
POWER = 4 * 30  # launches of the operator norm


@pytest.mark.parametrize("halpern", [False, True])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("iters", [1, 39])
def test_iterations_short_of_a_period(pkg, halpern, precision, iters):
    ps = [pkg.lpgen.random_equality_lp(*size, seed=70 + i) for i, size in enumerate(SIZES[precision])]
    misfit = pkg.lpgen.random_equality_lp(20000, 60000, 3, seed=9)
    rules = dict(termination_rule="relative_kkt_l2", restart_rule="adaptive_l2") if halpern else {}
    opt = pkg.PdhgOptions(max_iterations=iters, tolerance=1e-12, precision=precision, halpern=halpern, **rules)
    got = []
    for batch, launches in ((ps, len(ps)), (ps + [misfit], 2 * iters)):
        with pkg.Engine(0) as e:
            e.load_batch(batch)
            rs = e.solve_batch(opt)
        assert all(r.kernel_launches == POWER + launches + 2 for r in rs), rs[0].kernel_launches
        got.append(rs)
    eps = np.finfo(np.float32 if precision == "mixed" else np.float64).eps
    tol = iters * (64 if precision == "mixed" else 1500) * eps
    for p, a, b in zip(ps, *got):
        assert a.status == b.status == "iteration_limit" and a.iterations == b.iterations == iters
        assert np.any(a.primal) or np.any(a.dual)
        for u, v in ((a.primal, b.primal), (a.dual, b.dual)):
            assert np.max(np.abs(u - v)) <= tol * max(1.0, np.max(np.abs(v))), (p.m, p.n)
