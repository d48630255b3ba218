"""GP_FLAG_VERIFY on levels that one thread-block cluster refines: it checks what an ordinary call runs.

With the flag the cluster stops after every batch for the host to compare cut and cache, and goes on; the labels and
every statistic stay as they are without it.
"""
import numpy as np
import pytest

from graphs import launches_of, random_graph
from test_gpu_cluster_levels import mixed
from test_gpu_repair_sizes import FIELDS, overloaded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree,k,extra,weighted", [
    (700, 6, 5, 0, False), (9000, 6, 20, 0, True), (16384, 6, 8, 900, False), (16384, 6, 8, 900, True),
    (40000, 5, 4, 15000, True), (60000, 3, 8, 30000, False)])
def test_the_cluster_is_checked_after_every_batch(gp, ctx, oracle, n, degree, k, extra, weighted):
    g = random_graph(gp, n, degree, n + k, 9 if weighted else 0, 4 if weighted else 0)
    start = overloaded(n, k, extra, 3) if extra else mixed(n, k, 0.2, 3)
    eps = 1.15 if weighted else 1.04
    want, ostats = oracle.refine(g, start, k, eps)
    with launches_of(ctx, "k_refine_cluster") as ordinary:
        plain, pstats = ctx.refine(g, start, k, eps)
    with launches_of(ctx, "k_refine_cluster") as checked:
        labels, stats = ctx.refine(g, start, k, eps, flags=gp.FLAG_QUIET | gp.FLAG_VERIFY)
    np.testing.assert_array_equal(plain, want)
    np.testing.assert_array_equal(labels, want)
    for key in FIELDS:
        assert stats[key] == pstats[key] == ostats[key], key
    # A round's propagation is a batch, and so is every repair iteration that is not the last of a repair.
    assert ordinary[0] >= 1 and checked[0] >= ordinary[0] + stats["rounds"] - 2


def test_a_repair_that_cannot_succeed(gp, ctx):
    vw = np.ones(400, np.uint32)
    vw[:5] = 60
    g = random_graph(gp, 400, 4, 1)
    g = gp.Graph(g.offsets, g.neighbors, vw, g.edge_weights)
    start = (np.arange(400) % 5).astype(np.int32)
    start[:5] = 0
    for flags in (gp.FLAG_QUIET, gp.FLAG_QUIET | gp.FLAG_VERIFY):
        with pytest.raises(gp.GpartError) as e:
            ctx.refine(g, start, 5, 1.0, flags=flags)
        assert e.value.status == 2


def test_whole_partition(gp, ctx):
    for g, k in ((gp.grid2d(120, 90), 6), (gp.mesh3d(20, 20, 20, weighted=True, seed=2), 16)):
        plain, _ = ctx.partition(g, k, 1.03, 4)
        with launches_of(ctx, "k_refine_cluster") as checked:
            labels, _ = ctx.partition(g, k, 1.03, 4, gp.FLAG_QUIET | gp.FLAG_VERIFY)
        np.testing.assert_array_equal(labels, plain)
        assert checked[0] > 10
