"""Passes launched while the pass before still runs (pass.cuh) against the
same passes in full order: a traced solve copies the iterates out after every
iteration, so none of its primal passes starts early. Same arithmetic, so the
two must end in the same bits; a pass that read before its wait would not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RULES = dict(termination_rule="relative_kkt_l2", restart_rule="adaptive_l2",
             primal_weight_update=True, tolerance=1e-12, polish_iterations=0)
FORMS = {"exact": {}, "averaged": RULES, "halpern": dict(RULES, halpern=True)}
LPS = {
    "one_row": lambda L: L.random_equality_lp(1, 2, 1, seed=1),
    "columns_of_four": lambda L: L.random_equality_lp(60, 150, 4, seed=2),
    "block_edge": lambda L: L.random_equality_lp(171, 513, 3, seed=3),
    "columns_of_two": lambda L: L.transportation_lp(40, 83, seed=4),
    "columns_of_eight": lambda L: L.random_equality_lp(257, 771, 8, seed=5),
    "empty_and_long_rows": lambda L: L.badly_scaled_lp(500, 1200, 5, seed=6),
    "many_blocks": lambda L: L.random_equality_lp(30000, 70001, 7, seed=7),
    # thread rows of more than the held entries, warp rows around their rounds
    "row_tiers": lambda L: L.row_lengths_lp([0, 1, 7, 8, 9, 31, 32, 33, 127, 128, 129, 256, 257,
                                             511, 512, 513, 4097] * 2, 5000, seed=8),
}


@pytest.mark.parametrize("form,precision", [("exact", "fp64_exact"), ("averaged", "mixed"),
                                            ("averaged", "fp64"), ("halpern", "mixed"),
                                            ("halpern", "fp64")])
@pytest.mark.parametrize("name", sorted(LPS))
def test_early_passes_are_the_ordered_ones(pkg, name, form, precision):
    p = LPS[name](pkg.lpgen)
    kw = dict(FORMS[form], precision=precision)
    with pkg.Engine(0) as e:
        e.load(p)
        for iters in (80, 133):  # whole periods, and a last one cut short
            a = e.solve(pkg.PdhgOptions(max_iterations=iters, **kw))
            b = e.solve(pkg.PdhgOptions(max_iterations=iters, trace_iters=iters, **kw))
            assert (a.status, a.iterations, a.restarts) == (b.status, b.iterations, b.restarts)
            for f in ("primal", "dual", "reduced_costs"):
                np.testing.assert_array_equal(getattr(a, f), getattr(b, f))
            assert a.objective == b.objective
