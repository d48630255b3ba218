"""The capacity exchange with lists on both sides of what one block sorts (4096), against the oracle."""
import numpy as np
import pytest

from graphs import hubs_and_leaves, random_graph
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
