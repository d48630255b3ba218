"""Small symmetric graphs for the size tests, from edge lists."""
import contextlib

import numpy as np


def symmetric(gp, n, u, v, vw=None, seed=0, max_weight=0):
    """The graph of the undirected edges (u, v): no self loops or duplicates, rows sorted; edge weights 1..max_weight."""
    u, v = np.asarray(u, np.int64), np.asarray(v, np.int64)
    keep = u != v
    lo, hi = np.minimum(u, v)[keep], np.maximum(u, v)[keep]
    key = np.unique(lo * n + hi)
    lo, hi = key // n, key % n
    src, dst = np.concatenate([lo, hi]), np.concatenate([hi, lo])
    order = np.argsort(src * n + dst, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    ew = None
    if max_weight:
        w = np.random.default_rng(seed).integers(1, max_weight + 1, len(key)).astype(np.uint32)
        ew = np.concatenate([w, w])[order]
    return gp.Graph(off, dst[order].astype(np.int32), vw, ew)


def random_graph(gp, n, degree, seed, max_weight=0, vw_max=0):
    rng = np.random.default_rng(seed)
    m = n * degree // 2
    vw = rng.integers(1, vw_max + 1, n).astype(np.uint32) if vw_max else None
    return symmetric(gp, n, rng.integers(0, n, m), rng.integers(0, n, m), vw, seed, max_weight)


def hubs_and_leaves(gp, n, hubs, seed, max_weight=0):
    """Every vertex on two hubs, and a sparse random graph beneath."""
    rng = np.random.default_rng(seed)
    leaf = np.arange(n)
    u = np.concatenate([leaf, leaf, rng.integers(0, n, n)])
    v = np.concatenate([rng.integers(0, hubs, n), rng.integers(0, hubs, n), rng.integers(0, n, n)])
    return symmetric(gp, n, u, v, None, seed, max_weight)


@contextlib.contextmanager
def launches_of(ctx, kernel):
    """A list that holds, after the block, how often kernels of this name were started by the context's calls in it."""
    count = []
    ctx.profile_begin(kernel)
    try:
        yield count
    finally:
        count.append(ctx.profile_end()[0])
