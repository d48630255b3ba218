"""Coarsening and contraction at the sizes where another kernel takes over, against the oracle.

Coarse rows of up to 16 raw entries are sorted two to a warp; levels of 65,536 vertices and more are matched with 1, 8 or
32 lanes a row by their average row; up to 2048 requests of a round are ordered by one block; long rows are counted by
one block up to 49,152 targets, a segment of targets at a time above.
"""
import numpy as np
import pytest

from graphs import hubs_and_leaves, launches_of, random_graph, symmetric

pytestmark = pytest.mark.gpu


def check(gp, ctx, oracle, g, k, seed=0):
    want, cut = oracle.partition(g, k, 1.05, seed)
    got, stats = ctx.partition(g, k, 1.05, seed, gp.FLAG_QUIET | gp.FLAG_KEEP_HIERARCHY)
    expected = oracle.levels()
    levels = ctx.levels()
    assert len(levels) == len(expected)
    for mine, theirs in zip(levels, expected):
        for key in ("offsets", "neighbors", "edge_weights", "vertex_weights", "map"):
            if theirs[key] is not None:
                np.testing.assert_array_equal(mine[key], theirs[key], err_msg=key)
    assert stats.edge_cut == cut
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("degree", [1, 2, 4, 5, 7, 8, 9, 15, 16, 17])
def test_regular_rows(gp, ctx, oracle, degree):
    """Circulant graphs: two fine rows make a raw coarse row of twice the degree, around the class edges."""
    n = 3001
    i = np.arange(n)
    u = np.concatenate([i] * ((degree + 1) // 2))
    v = np.concatenate([(i + d * d + d) % n for d in range(1, (degree + 1) // 2 + 1)])
    check(gp, ctx, oracle, symmetric(gp, n, u, v, None, degree, 5), 4)


@pytest.mark.parametrize("n,hubs", [(1500, 20), (2600, 3), (5200, 40), (9000, 9), (40000, 300)])
@pytest.mark.parametrize("weight", [0, 7])
def test_ordered_requests(gp, ctx, oracle, n, hubs, weight):
    """Leaves that ask for few receivers: from a handful to far more than one block orders."""
    check(gp, ctx, oracle, hubs_and_leaves(gp, n, hubs, n, weight), 8, 3)


@pytest.mark.parametrize("n,hubs", [(60000, 5), (110000, 5), (150000, 6), (450000, 9)])
def test_long_coarse_rows(gp, ctx, oracle, n, hubs):
    check(gp, ctx, oracle, hubs_and_leaves(gp, n, hubs, n, 3), 4, 2)


@pytest.mark.parametrize("n,degree", [(65535, 12), (65536, 6), (65536, 12), (70001, 40)])
def test_matching_levels(gp, ctx, oracle, n, degree):
    check(gp, ctx, oracle, random_graph(gp, n, degree, degree, 4, 3), 6, 1)


def test_isolated_and_empty(gp, ctx, oracle):
    rng = np.random.default_rng(5)
    u, v = rng.integers(0, 700, 1500), rng.integers(0, 700, 1500)
    check(gp, ctx, oracle, symmetric(gp, 6000, u, v), 4)


@pytest.mark.parametrize("build,taken,absent", [
    (lambda gp: random_graph(gp, 65536, 6, 6, 4, 3), ["k_match_choose<1>", "k_sort_rows_short"], ["k_dense_rows"]),
    (lambda gp: random_graph(gp, 65536, 12, 12, 4, 3), ["k_match_choose<8>"], ["k_match_choose<32>"]),
    (lambda gp: random_graph(gp, 70001, 40, 40, 4, 3), ["k_match_choose<32>"], ["k_match_choose<8>"]),
    (lambda gp: hubs_and_leaves(gp, 2600, 3, 2600), ["k_order_block<false>", "k_order_block<true>"],
     ["k_ordered_accept", "k_pair_flags"]),
    (lambda gp: hubs_and_leaves(gp, 40000, 300, 40000), ["k_order_block<false>", "k_ordered_accept", "k_pair_flags"], []),
    (lambda gp: hubs_and_leaves(gp, 60000, 5, 60000, 3), ["k_dense_rows"], ["k_dense_pieces", "k_large_records"]),
    (lambda gp: hubs_and_leaves(gp, 450000, 9, 450000, 3), ["k_dense_rows", "k_dense_pieces", "k_dense_copy"],
     ["k_large_records"])])
def test_the_named_kernels_run(gp, ctx, build, taken, absent):
    g = build(gp)
    for kernel in taken + absent:
        with launches_of(ctx, kernel) as started:
            ctx.partition(g, 6, 1.05, 1)
        assert (started[0] > 0) == (kernel in taken), kernel


def test_long_rows_with_zero_weights_are_sorted(gp, ctx, oracle):
    """A counter cannot tell a target of weight zero from an absent one: the sorts take such levels' long rows."""
    g = hubs_and_leaves(gp, 60000, 5, 60000, 3)
    g = gp.Graph(g.offsets, g.neighbors, g.vertex_weights, g.edge_weights - 1)
    assert (g.edge_weights == 0).any()
    check(gp, ctx, oracle, g, 4, 2)
    for kernel in ("k_large_records", "k_dense_rows"):
        with launches_of(ctx, kernel) as started:
            ctx.partition(g, 4, 1.05, 2)
        assert (started[0] > 0) == (kernel == "k_large_records")
