"""Capacity repair at the lengths of its donor list where another path takes over.

A list of up to 2048 donors is ordered and placed by one block, a longer one by the device-wide path, and after a long
list the next one's length is read first.  Two parts that overflow by a chosen weight, over edges that leave most donors
in few gain classes, make lists on both sides; the oracle says what the labels and every statistic have to be.
"""
import numpy as np
import pytest

from graphs import launches_of, random_graph

pytestmark = pytest.mark.gpu
FIELDS = ("rounds", "admission_iterations", "checkpoint_updates", "proposals", "accepted", "initial_cut", "final_cut",
          "final_max_part_weight", "lp_cut_gain", "lp_cut_loss", "rebalance_cut_gain", "rebalance_cut_loss",
          "group_cut_gain", "group_accepted")


def overloaded(n, k, extra, seed):
    """Equal blocks, then `extra` vertices of the other parts moved to parts 0 and 1."""
    rng = np.random.default_rng(seed)
    labels = (np.arange(n) * k // n).astype(np.int32)
    others = rng.permutation(np.flatnonzero(labels > 1))[:extra]
    labels[others] = others % 2
    return labels


def check(gp, ctx, oracle, g, start, k, eps, rounds=32):
    want, ostats = oracle.refine(g, start, k, eps, rounds, 2)
    got, stats = ctx.refine(g, start, k, eps, rounds, 2)
    np.testing.assert_array_equal(got, want)
    for key in FIELDS:
        assert stats[key] == ostats[key], key


@pytest.mark.parametrize("n,degree,k,extra", [
    (600, 4, 3, 60), (5000, 0, 4, 1500), (5000, 3, 4, 2300), (16384, 6, 8, 2040), (16384, 6, 8, 2060),
    (40000, 0, 16, 9000), (40000, 8, 128, 12000), (65536, 4, 5, 30000), (65537, 4, 5, 30000), (90000, 5, 40, 700),
    (90000, 5, 40, 40000)])
@pytest.mark.parametrize("weighted", [False, True])
def test_repair_equals_the_oracle(gp, ctx, oracle, n, degree, k, extra, weighted):
    g = random_graph(gp, n, degree, n + extra, 9 if weighted else 0, 5 if weighted else 0)
    check(gp, ctx, oracle, g, overloaded(n, k, extra, k), k, 1.05 if not weighted else 1.10, 6)


def test_repair_without_a_cache(gp, ctx, oracle):
    """A mesh whose rows are short next to k recomputes affinities; both list lengths."""
    g = gp.mesh3d(50, 45, 41, weighted=True, seed=3)
    for extra in (300, 20000):
        check(gp, ctx, oracle, g, overloaded(g.n, 100, extra, 1), 100, 1.05, 4)


@pytest.mark.parametrize("n,degree,k,vw_max,eps", [
    (3000, 0, 3, 200, 1.03), (3000, 0, 33, 200, 1.05), (3000, 2, 128, 12, 1.20), (40000, 1, 128, 200, 1.03),
    (70000, 0, 128, 3000, 1.01), (70000, 2, 32, 3000, 1.002)])
def test_tickets_over_parts_that_fit(gp, ctx, oracle, n, degree, k, vw_max, eps):
    """Donors without a neighbour elsewhere, many heavier than the room of some or of all parts."""
    g = random_graph(gp, n, degree, n + k, 3, vw_max)
    check(gp, ctx, oracle, g, overloaded(n, k, n // 5, k), k, eps, 6)


@pytest.mark.parametrize("n,degree,k,extra,weighted,short,long", [
    (90000, 5, 40, 700, False, True, True), (90000, 5, 40, 700, True, True, False),
    (40000, 8, 128, 12000, False, False, True), (40000, 0, 16, 9000, False, False, True)])
def test_both_paths_are_taken(gp, ctx, n, degree, k, extra, weighted, short, long):
    """Iterations whose list one block places and iterations whose list goes through the device-wide path."""
    g = random_graph(gp, n, degree, n + extra, 9 if weighted else 0, 5 if weighted else 0)
    start = overloaded(n, k, extra, k)
    took = {}
    for kernel in ("k_repair_block", "k_repair_active", "k_repair_bounds"):
        with launches_of(ctx, kernel) as started:
            ctx.refine(g, start, k, 1.10 if weighted else 1.05, 6, 2)
        took[kernel] = started[0]
    assert (took["k_repair_active"] > 0) == long
    assert (took["k_repair_bounds"] > took["k_repair_active"]) == short  # one launch an iteration
    assert took["k_repair_block"] > 0  # offered the first list whatever its length


def test_both_paths_without_a_cache(gp, ctx):
    g = gp.mesh3d(50, 45, 41, weighted=True, seed=3)
    for extra, long in ((300, False), (20000, True)):
        with launches_of(ctx, "k_repair_dest_od") as iterations:
            ctx.refine(g, overloaded(g.n, 100, extra, 1), 100, 1.05, 4, 2)
        with launches_of(ctx, "k_repair_active") as long_lists:
            ctx.refine(g, overloaded(g.n, 100, extra, 1), 100, 1.05, 4, 2)
        assert (long_lists[0] > 0) == long and iterations[0] > long_lists[0]
