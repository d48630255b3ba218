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


def stuck_pairs(gp, n, k, light_max, seed):
    """A graph and labels whose first round cannot be repaired, which leaves everything to the exchange: every light
    vertex (weight 1..light_max) is drawn to the other part of its pair (p, p ^ 1), and each part holds a heavy vertex
    that is drawn there as well and does not fit.  Two strong edges a vertex across, three weak ones within the part."""
    rng = np.random.default_rng(seed)
    vertex = np.arange(n)
    across, within = np.repeat(vertex, 2), np.repeat(vertex, 3)
    there = rng.integers(0, n // k, len(across)) * k + (across % k ^ 1)
    here = rng.integers(0, n // k, len(within)) * k + within % k
    heavy = n + np.arange(k)
    u, v = np.concatenate([across, within, heavy[0::2]]), np.concatenate([there, here, heavy[1::2]])
    weight = np.concatenate([np.full(len(across), 9), np.full(len(within), 1), np.full(k // 2, 10**6)])
    labels = np.concatenate([vertex % k, np.arange(k)]).astype(np.int32)
    total = n + k
    keep = u != v
    key, first = np.unique(np.minimum(u, v)[keep] * total + np.maximum(u, v)[keep], return_index=True)
    weight = weight[keep][first]
    src, dst = np.concatenate([key // total, key % total]), np.concatenate([key % total, key // total])
    order = np.argsort(src * total + dst, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=total))]).astype(np.int32)
    vw = np.concatenate([rng.integers(1, light_max + 1, n), np.zeros(k)]).astype(np.uint32)
    loads = np.bincount(labels, weights=vw, minlength=k).astype(np.uint32)
    vw[n:] = loads.max() * 5 // 2 - loads
    return gp.Graph(off, dst[order].astype(np.int32), vw, np.concatenate([weight, weight])[order].astype(np.uint32)), labels


@contextlib.contextmanager
def launches_of(ctx, kernel):
    """A list that holds, after the block, how often kernels of this name were started by the context's calls in it."""
    count = []
    ctx.profile_begin(kernel)
    try:
        yield count
    finally:
        count.append(ctx.profile_end()[0])
