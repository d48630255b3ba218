"""Levels refined by one thread-block cluster, at the sizes where it can go wrong.

A cluster takes levels of up to 65,536 vertices, 2^19 cache cells, 2^18 entries and 16 entries a row, 8192 vertices a
pass; rows above 256 entries are done by a whole block, up to 512 of them a pass.  The oracle says what the labels and
every statistic have to be.
"""
import numpy as np
import pytest

from graphs import hubs_and_leaves, launches_of, random_graph, symmetric
from test_gpu_repair_sizes import check, overloaded

pytestmark = pytest.mark.gpu


def mixed(n, k, share, seed):
    rng = np.random.default_rng(seed)
    labels = (np.arange(n) * k // n).astype(np.int32)
    some = rng.permutation(n)[: max(2, int(n * share))]
    labels[some] = labels[np.roll(some, 1)]
    return labels


def check_path(gp, ctx, oracle, g, start, k, eps, rounds=32):
    """check(), and that the cluster took the level if and only if its rule says so; how often it was started."""
    with launches_of(ctx, "k_refine_cluster") as started:
        check(gp, ctx, oracle, g, start, k, eps, rounds)
    assert (started[0] > 0) == (g.n <= 65536 and g.n * k <= 1 << 19 and g.m <= min(1 << 18, 16 * g.n))
    return started[0]


@pytest.mark.parametrize("n,k", [(300, 2), (511, 7), (512, 9), (513, 20), (8191, 64), (8192, 63), (8192, 65), (8193, 37),
                                 (40000, 13), (40000, 14), (65535, 3), (65536, 2), (65537, 2)])
@pytest.mark.parametrize("weighted", [False, True])
def test_passes(gp, ctx, oracle, n, k, weighted):
    g = random_graph(gp, n, 4 if n > 60000 else 6, n + k, 9 if weighted else 0, 4 if weighted else 0)
    check_path(gp, ctx, oracle, g, mixed(n, k, 0.2, k), k, 1.05 if not weighted else 1.2)


@pytest.mark.parametrize("n,hubs", [(4000, 1), (4000, 12), (30000, 75), (40000, 300)])
def test_long_rows(gp, ctx, oracle, n, hubs):
    g = hubs_and_leaves(gp, n, hubs, hubs, 5)
    assert (np.diff(g.offsets) > 256).any()
    check_path(gp, ctx, oracle, g, mixed(n, 9, 0.3, 1), 9, 1.06)


def test_more_long_rows_than_a_block_sets_aside(gp, oracle):
    """1024 rows of about 110 entries in the first block's share, long ones by this context's threshold."""
    n = 20000
    rng = np.random.default_rng(8)
    rows = np.repeat(np.concatenate([np.arange(512), np.arange(8192, 8704)]), 110)
    g = symmetric(gp, n, rows, rng.integers(0, n, len(rows)))
    assert g.m <= 1 << 18 and g.m <= 16 * n
    with gp.Context(0) as own:
        own.set_option("refine_heavy_small", 64)
        check_path(gp, own, oracle, g, mixed(g.n, 9, 0.5, 1), 9, 1.06, 3)


@pytest.mark.parametrize("n,degree", [(16384, 15), (16384, 17), (9000, 15), (9000, 17)])  # about 2^18 entries, 16 a row
def test_entry_limits(gp, ctx, oracle, n, degree):
    g = random_graph(gp, n, degree, degree)
    check_path(gp, ctx, oracle, g, mixed(g.n, 12, 0.1, 2), 12, 1.03, 5)


@pytest.mark.parametrize("k", [2, 3, 127, 128])
def test_part_counts(gp, ctx, oracle, k):
    g = random_graph(gp, 4000, 8, k, 3, 3)
    check_path(gp, ctx, oracle, g, overloaded(g.n, k, 600, 4), k, 1.10)


@pytest.mark.parametrize("n,hubs,k", [(20000, 60, 4), (20000, 60, 16), (40000, 20, 4)])
def test_resumed_after_a_round(gp, ctx, oracle, n, hubs, k):
    """The parts fit at the start, then a round moves thousands of leaves to the hubs' part: its repair lists more donors
    than one block takes, so the host completes it and starts the cluster again behind it."""
    g = hubs_and_leaves(gp, n, hubs, 2, 4)
    start = mixed(n, k, 0.0001, 1)
    assert np.bincount(start).max() <= n * 1.03 // k
    assert check_path(gp, ctx, oracle, g, start, k, 1.03) > 1


def test_resumed_after_the_initial_repair(gp, ctx, oracle):
    g = random_graph(gp, 5000, 3, 7300)
    start = overloaded(5000, 4, 2300, 4)
    assert check_path(gp, ctx, oracle, g, start, 4, 1.05, 6) > 1
    with launches_of(ctx, "k_repair_active") as long_lists:
        ctx.refine(g, start, 4, 1.05, 6)
    assert long_lists[0] > 0


@pytest.mark.parametrize("rounds", [0, 1, 64])
def test_round_budgets(gp, ctx, oracle, rounds):
    g = gp.grid2d(70, 61)
    check_path(gp, ctx, oracle, g, mixed(g.n, 6, 0.1, 3), 6, 1.03, rounds)


def test_repair_that_cannot_succeed(gp, ctx, oracle):
    """Heavy vertices in a part they overflow and no part with room for them."""
    vw = np.ones(400, np.uint32)
    vw[:5] = 60
    g = random_graph(gp, 400, 4, 1)
    g = gp.Graph(g.offsets, g.neighbors, vw, g.edge_weights)
    start = (np.arange(400) % 5).astype(np.int32)
    start[:5] = 0
    with pytest.raises(gp.GpartError) as mine:
        ctx.refine(g, start, 5, 1.0)
    assert mine.value.status == 2
    with pytest.raises(Exception):
        oracle.refine(g, start, 5, 1.0)
