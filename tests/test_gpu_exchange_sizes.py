"""The capacity exchange, whose lists one block per part sorts, against the oracle.

A part's lists hold at most 2048 fragments and 4608 moves; the oracle says how long the longest were.
"""
import numpy as np
import pytest

from graphs import hubs_and_leaves, random_graph, stuck_pairs
from test_gpu_cluster_levels import mixed
from test_gpu_repair_sizes import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree,k", [(500, 4, 4), (3000, 6, 16), (20000, 4, 32), (60000, 3, 64), (65536, 6, 128),
                                        (65536, 3, 40)])
@pytest.mark.parametrize("weighted", [False, True])
def test_exchange(gp, ctx, oracle, n, degree, k, weighted):
    g = random_graph(gp, n, degree, n + k, 9 if weighted else 0, 3 if weighted else 0)
    check(gp, ctx, oracle, g, mixed(n, k, 0.05, k), k, 1.04 if not weighted else 1.15, 1)


def test_exchange_with_hubs(gp, ctx, oracle):
    g = hubs_and_leaves(gp, 30000, 60, 2, 4)
    check(gp, ctx, oracle, g, mixed(g.n, 24, 0.1, 5), 24, 1.05, 2)


@pytest.mark.parametrize("n,k,lights,slack", [(20000, 2, 1, 2), (20000, 2, 5, 0), (40000, 32, 1, 3), (40000, 32, 50, 8)])
def test_lists_at_their_bounds(gp, ctx, oracle, n, k, lights, slack):
    g, start = stuck_pairs(gp, n, k, lights, 1)
    check(gp, ctx, oracle, g, start, k, 1 + slack * k / int(g.vertex_weights.sum()) + 1e-9, 1)
    fragments, moves = oracle.exchange_lists()
    assert fragments == 2048 and moves > 2048
