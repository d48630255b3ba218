"""Performance cases: the calls a user of this partitioner makes, over their real range.

A case names one public call (``call``) and the graph(s) it works on:

``partition``  ``Context.partition_device``: the whole V-cycle on a graph resident in device memory, labels written to
               device memory (the headline call).
``host``       ``Context.partition``: the same from host arrays, upload and label download inside the call (what the
               command-line tool and a CPU program do).
``batch``      ``Context.partition_batch``: many uneven host graphs at once on one GPU.
``refine``     ``Context.refine``: one level of refinement of a caller's labels (host arrays in and out).
``evaluate``   ``Context.evaluate_device``: cut and part loads of device labels, waits for the result.
``static``     ``evaluate_device_static``: its allocation-free twin, which does not wait.

Graph families: ``grid`` (2D five-point, n = x*y), ``mesh`` (3D seven-point, n = x*y*z) and ``rmat`` (edge factor 8..16,
a=.57 b=.19 c=.19, symmetrised, self loops and duplicates removed, rows sorted; any n, odd ones included).  Weighted
graphs carry uniform vertex weights in [1, vw] and symmetric uniform edge weights in [1, ew].

Inputs come from the seed alone: the R-MAT samples, the weights, the start labels, and the partitioner's own seed
argument.  All outputs are integers and have to be equal.
"""
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """This repository's package (its folder's name is not an identifier), from the working tree first."""
    if "acc_gp_b200" in sys.modules:
        return sys.modules["acc_gp_b200"]
    for root in (os.getcwd(), _ROOT):
        folder = os.path.join(root, "acc-gp_b200")
        if os.path.exists(os.path.join(folder, "__init__.py")):
            break
    spec = importlib.util.spec_from_file_location("acc_gp_b200", os.path.join(folder, "__init__.py"),
                                                  submodule_search_locations=[folder])
    module = importlib.util.module_from_spec(spec)
    sys.modules["acc_gp_b200"] = module
    spec.loader.exec_module(module)
    return module


gp = _package()
_context = None


def _ctx():
    """The one context that a program with one host thread keeps for all its graphs."""
    global _context
    if _context is None:
        _context = gp.Context(0)
    return _context


def listed():
    return [
        # The headline: a large skewed graph, unit weights, resident in device memory.
        dict(name="rmat22_k64", call="partition", family="rmat", n=1 << 22, factor=16, vw=1, ew=1, k=64, eps=1.03),
        # A large simulation mesh with weights, at the largest part count.
        dict(name="mesh256w_k128", call="partition", family="mesh", x=256, y=256, z=256, vw=4, ew=16, k=128, eps=1.03),
        # An ordinary small grid: a chain of short kernels and host decisions.
        dict(name="grid256_k8", call="partition", family="grid", x=256, y=256, vw=1, ew=1, k=8, eps=1.03),
        # The smallest graph of the batched workload, alone: latency only.
        dict(name="grid33x31_k4", call="partition", family="grid", x=33, y=31, vw=1, ew=1, k=4, eps=1.03),
        # Serving requests: weighted skewed graphs of a resident pool, any k, tight and loose balance; odd sizes.
        dict(name="rmat300007w_k37", call="partition", family="rmat", n=300007, factor=12, vw=16, ew=64, k=37, eps=1.01),
        dict(name="rmat32768w_k93", call="partition", family="rmat", n=32768, factor=12, vw=16, ew=64, k=93, eps=1.05),
        # A program whose graph is in host memory: an odd-sized mesh, unit weights.
        dict(name="host_mesh101x97x103_k32", call="host", family="mesh", x=101, y=97, z=103, vw=1, ew=1, k=32, eps=1.03),
        # The batched form: uneven graphs, half skewed and half grids and meshes.
        dict(name="batch24", call="batch", count=24, low=1000, high=200000, concurrency=8, eps=1.03),
        # Refinement of a caller's labels, on a mesh and on a skewed graph.
        dict(name="refine_mesh64w_k32", call="refine", family="mesh", x=64, y=64, z=64, vw=4, ew=16, k=32, eps=1.03,
             swapped=0.03),
        dict(name="refine_rmat100003_k16", call="refine", family="rmat", n=100003, factor=16, vw=1, ew=1, k=16, eps=1.05,
             swapped=0.08),
        # Judging a labelling: of the headline graph, and of a small grid inside somebody's own loop.
        dict(name="evaluate_rmat22_k64", call="evaluate", family="rmat", n=1 << 22, factor=16, vw=1, ew=1, k=64,
             swapped=0.08),
        dict(name="static_grid256_k8", call="static", family="grid", x=256, y=256, vw=4, ew=16, k=8, swapped=0.03),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _parts(rng, n):
    """A part count in 2..128 that leaves every part at least 200 vertices."""
    return max(2, min(_log_int(rng, 2, 128), n // 200))


def _family(rng, low, high):
    """A graph of about low..high vertices (log-uniform): half skewed, half grids and meshes, half of each weighted."""
    n = _log_int(rng, low, high)
    vw, ew = rng.choice([(1, 1), (1, 1), (4, 16), (16, 64)])
    pick = rng.random()
    if pick < 0.5:
        n = n if rng.random() < 0.6 else 1 << round(math.log2(n))
        return dict(family="rmat", n=n, factor=rng.randint(8, 16), vw=vw, ew=ew)
    if pick < 0.75:
        x = max(8, int(n ** 0.5 * rng.uniform(0.6, 1.6)))
        return dict(family="grid", x=x, y=max(8, n // x), vw=vw, ew=ew)
    x = max(6, int(n ** (1 / 3) * rng.uniform(0.7, 1.4)))
    y = max(6, int(n ** (1 / 3) * rng.uniform(0.7, 1.4)))
    return dict(family="mesh", x=x, y=y, z=max(4, n // (x * y)), vw=vw, ew=ew)


def draw(rng):
    call = rng.choice(["partition"] * 5 + ["host", "refine", "evaluate", "static", "batch"])
    if call == "batch":
        return dict(call=call, count=rng.randint(6, 32), low=1000, high=_log_int(rng, 20000, 300000),
                    concurrency=rng.choice([4, 8, 16]), eps=1.03)
    case = dict(call=call, **_family(rng, 1000, 3000000 if call in ("partition", "evaluate") else 600000))
    k = _parts(rng, _vertices(case))
    if call in ("evaluate", "static"):
        return dict(case, k=k, swapped=rng.choice([0.03, 0.08]))
    # A tight balance needs parts of some size: floor(total * eps / k) * k has to hold the total.
    eps = rng.choice([1.01, 1.03, 1.05])
    if call == "refine":
        return dict(case, k=k, eps=max(1.03, eps), swapped=rng.choice([0.03, 0.08]))
    return dict(case, k=k, eps=eps)


# ---------------------------------------------------------------- inputs


def _vertices(case):
    if case["family"] == "rmat":
        return case["n"]
    return case["x"] * case["y"] * case.get("z", 1)


def _edges(case):
    """Directed CSR entries; for R-MAT (whose number depends on the seed) the samples less about a tenth."""
    if case["family"] == "rmat":
        return int(1.85 * case["factor"] * case["n"])
    x, y, z = case["x"], case["y"], case.get("z", 1)
    return 2 * ((x - 1) * y * z + x * (y - 1) * z + x * y * (z - 1))


def _rmat(n, factor, gen, device):
    bits = max(1, (n - 1).bit_length())
    samples = factor * n
    src = torch.zeros(samples, dtype=torch.int32, device=device)
    dst = torch.zeros(samples, dtype=torch.int32, device=device)
    u = torch.empty(samples, dtype=torch.float32, device=device)
    for _ in range(bits):
        u.uniform_(generator=gen)
        down = u >= 0.76                                  # c or d: the source's bit
        right = ((u >= 0.57) & ~down) | (u >= 0.95)       # b or d: the target's bit
        src.mul_(2).add_(down)
        dst.mul_(2).add_(right)
    keep = (src != dst) & (src < n) & (dst < n)
    src, dst = src[keep].long(), dst[keep].long()
    keys = torch.unique(torch.cat([src * n + dst, dst * n + src]))
    del src, dst, u, keep
    rows = torch.div(keys, n, rounding_mode="floor")
    neighbors = (keys - rows * n).int()
    return rows, neighbors


def _lattice(x, y, z, device):
    """The seven-point mesh, id = i + x*(j + y*l), rows sorted."""
    n = x * y * z
    v = torch.arange(n, dtype=torch.int32, device=device)
    i, j, l = v % x, (v // x) % y, v // (x * y)
    steps = [(l > 0, -x * y), (j > 0, -x), (i > 0, -1), (i < x - 1, 1), (j < y - 1, x), (l < z - 1, x * y)]
    has = torch.stack([s[0] for s in steps], dim=1)
    to = torch.stack([v + s[1] for s in steps], dim=1)
    return has.sum(1), to[has].contiguous()


def _mix(a):
    """A 63-bit mix of int64 values (splitmix64's finaliser, logical shifts spelled out)."""
    for shift, mul in ((30, -0x40A7B892E31B1A47), (27, -0x6B2FB644ECCEEE15)):
        a = (a ^ ((a >> shift) & ((1 << (64 - shift)) - 1))) * mul
    return (a ^ ((a >> 31) & ((1 << 33) - 1))) & 0x7FFFFFFFFFFFFFFF


def _graph(case, gen, device):
    """offsets, neighbors, vertex weights, edge weights (device tensors; None for unit weights)."""
    n = _vertices(case)
    if case["family"] == "rmat":
        rows, neighbors = _rmat(n, case["factor"], gen, device)
        degree = torch.bincount(rows, minlength=n)
    else:
        degree, neighbors = _lattice(case["x"], case["y"], case.get("z", 1), device)
        rows = None
    offsets = torch.zeros(n + 1, dtype=torch.int32, device=device)
    offsets[1:] = torch.cumsum(degree, 0)
    vw = ew = None
    if case["vw"] > 1:
        vw = torch.randint(1, case["vw"] + 1, (n,), generator=gen, device=device, dtype=torch.int32)
    if case["ew"] > 1:
        if rows is None:
            rows = torch.repeat_interleave(torch.arange(n, device=device), degree)
        salt = int(torch.randint(0, 1 << 40, (1,), generator=gen, device=device))
        other = neighbors.long()
        key = torch.minimum(rows, other) * n + torch.maximum(rows, other)
        ew = (_mix(key + salt) % case["ew"] + 1).int()
    return offsets, neighbors, vw, ew


def _start_labels(case, gen, device):
    """k blocks of consecutive vertices, a share of which changed places with others: a labelling to judge or refine."""
    n, k = _vertices(case), case["k"]
    labels = (torch.arange(n, device=device) * k // n).int()
    some = torch.randperm(n, generator=gen, device=device)[: max(2, int(n * case["swapped"]))]
    labels[some] = labels[some.roll(1)]
    return labels


def _host(t, kind):
    return None if t is None else t.cpu().numpy().astype(kind, copy=False)


def _host_graph(arrays):
    return gp.Graph(_host(arrays[0], np.int32), _host(arrays[1], np.int32), _host(arrays[2], np.uint32),
                    _host(arrays[3], np.uint32))


def _batch_cases(case):
    """The batch's graphs: n log-uniform, even ones R-MAT, odd ones grids and meshes, k one of 4..128 where it fits.
    The seed makes what is in them, not how large they are."""
    rng = random.Random("batch %d %d %d" % (case["count"], case["low"], case["high"]))
    out = []
    for i in range(case["count"]):
        n = int(case["low"] * (case["high"] / case["low"]) ** ((i + rng.random()) / case["count"]))
        k = rng.choice([4, 8, 16, 32, 64, 128])
        while k > 2 and n < 200 * k:
            k //= 2
        if i % 2 == 0:
            g = dict(family="rmat", n=n, factor=rng.randint(8, 16))
        elif i % 4 == 1:
            x = int(n ** 0.5)
            g = dict(family="grid", x=x, y=n // x)
        else:
            x = int(n ** (1 / 3))
            g = dict(family="mesh", x=x, y=x, z=n // (x * x))
        out.append(dict(g, vw=1, ew=1, k=k))
    return out


class State:
    """What a program has in hand before the call."""


def prepare(case, seed):
    device = torch.device("cuda", 0)
    gen = torch.Generator(device=device)
    gen.manual_seed(1000003 * int(seed) + 17)
    s = State()
    s.case, s.ctx, s.seed = case, _ctx(), int(seed)
    if case["call"] == "batch":
        s.jobs = [(_host_graph(_graph(c, gen, device)), c["k"], case["eps"], s.seed) for c in _batch_cases(case)]
        return s
    s.arrays = _graph(case, gen, device)
    s.n, s.m = s.arrays[0].numel() - 1, s.arrays[1].numel()
    if case["call"] in ("host", "refine"):
        s.graph = _host_graph(s.arrays)
        s.arrays = None
    if case["call"] == "refine":
        s.labels = _host(_start_labels(case, gen, device), np.int32)
    elif case["call"] in ("evaluate", "static"):
        s.labels = _start_labels(case, gen, device)
        s.cut = torch.zeros(1, dtype=torch.int64, device=device)
        s.loads = torch.zeros(case["k"], dtype=torch.int64, device=device)
    elif case["call"] == "partition":
        s.labels = torch.empty(s.n, dtype=torch.int32, device=device)
    if s.arrays is not None:
        s.pointers = [None if t is None else t.data_ptr() for t in s.arrays]
    return s


def _verdict(stats):
    return [stats.edge_cut, stats.max_part_weight, stats.capacity, stats.initial_cut, stats.levels, stats.coarsest_vertices]


def run(state):
    s, case = state, state.case
    call = case["call"]
    if call == "partition":
        off, nbr, vw, ew = s.pointers
        stats = s.ctx.partition_device(off, nbr, s.n, s.m, vw, ew, case["k"], case["eps"], s.seed, s.labels.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream)
        return {"labels": s.labels, "verdict": _verdict(stats)}
    if call == "host":
        labels, stats = s.ctx.partition(s.graph, case["k"], case["eps"], s.seed)
        return {"labels": labels, "verdict": _verdict(stats)}
    if call == "batch":
        done = s.ctx.partition_batch(s.jobs, concurrency=case["concurrency"])
        return {"labels": [labels for labels, _, _ in done],
                "verdict": np.array([_verdict(stats) for _, stats, _ in done], np.int64)}
    if call == "refine":
        labels, stats = s.ctx.refine(s.graph, s.labels, case["k"], case["eps"])
        return {"labels": labels, "moves": [v for key, v in sorted(stats.items()) if key not in ("seconds", "kernel_launches")]}
    off, nbr, vw, ew = s.pointers
    evaluate = s.ctx.evaluate_device if call == "evaluate" else gp.evaluate_device_static
    evaluate(off, nbr, s.n, s.m, vw, ew, s.labels.data_ptr(), case["k"], s.cut.data_ptr(), s.loads.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
    return {"cut": s.cut, "loads": s.loads}


def work(case):
    """The CSR read once and the labels written once (read, when they are judged); each entry compared or added once."""
    if case["call"] == "batch":
        parts = [work(dict(c, call="host")) for c in _batch_cases(case)]
        return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}
    n, m = _vertices(case), _edges(case)
    size = 4 * (n + 1) + 4 * m + (4 * n if case["vw"] > 1 else 0) + (4 * m if case["ew"] > 1 else 0) + 4 * n
    if case["call"] == "refine":
        size += 4 * n
    if case["call"] in ("evaluate", "static"):
        size += 8 * (1 + case["k"])
    return {"bytes": size, "flops": m}


def tolerance(case):
    return "exact"


def exact(case, seed):
    """Cut and part loads in plain torch; a partition has no closed form."""
    if case["call"] not in ("evaluate", "static"):
        return None
    s = prepare(case, seed)
    off, nbr, vw, ew = s.arrays
    rows = torch.repeat_interleave(torch.arange(s.n, device=off.device), (off[1:] - off[:-1]).long())
    crossing = s.labels[rows] != s.labels[nbr.long()]
    cut = (crossing.long() if ew is None else crossing * ew.long()).sum() // 2
    weight = torch.ones(s.n, dtype=torch.int64, device=off.device) if vw is None else vw.long()
    loads = torch.zeros(case["k"], dtype=torch.int64, device=off.device).index_add_(0, s.labels.long(), weight)
    return {"cut": cut.reshape(1), "loads": loads}
