"""The evaluation kernels at the sizes where their split of the work can go wrong.

A warp reads 256 entries and the ends of 32 rows a step, and all warps share the merged sequence of rows and entries
evenly: hub rows, stretches of empty rows, rows that end on a window's edge, and graphs smaller than one share.  The
results are integers and have to equal a plain numpy count.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def degrees(shape, rng):
    return {
        "one_empty": np.zeros(1, np.int64),
        "one_row": np.array([700]),
        "row_ends_at_256": np.array([256, 256, 255, 1, 0, 0, 257, 512, 31, 1]),
        "empty_head_and_tail": np.concatenate([np.zeros(5000, np.int64), [3, 0, 0, 900], np.zeros(70000, np.int64)]),
        "hub_last": np.concatenate([np.ones(40000, np.int64), [300000]]),
        "hub_first": np.concatenate([[300000], np.zeros(40000, np.int64)]),
        "many_hubs": rng.choice([0, 1, 2, 31, 32, 33, 255, 256, 257, 3000], 4000),
        "short": rng.integers(0, 5, 300001),
    }[shape]


@pytest.mark.parametrize("shape", ["one_empty", "one_row", "row_ends_at_256", "empty_head_and_tail", "hub_last",
                                   "hub_first", "many_hubs", "short"])
@pytest.mark.parametrize("k,weighted", [(1, False), (7, True), (128, True)])
def test_cut_and_loads_equal_a_plain_count(gp, ctx, shape, k, weighted):
    import torch
    rng = np.random.default_rng(len(shape) * 131 + k)
    deg = degrees(shape, rng)
    n, m = len(deg), int(deg.sum())
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    nbr = rng.integers(0, n, m).astype(np.int32)
    vw = rng.integers(1, 2**32, n, dtype=np.uint32) if weighted else None
    ew = rng.integers(0, 2**32, m, dtype=np.uint32) if weighted else None
    # Half the labels in blocks (warps of one label), half of them anything.
    labels = (np.arange(n) * k // n).astype(np.int32)
    mixed = rng.random(n) < 0.5 if k > 1 else np.zeros(n, bool)
    mixed[: n // 2] = False
    labels[mixed] = rng.integers(0, k, int(mixed.sum()))
    crossing = labels[np.repeat(np.arange(n), deg)] != labels[nbr]
    cut = int((crossing if ew is None else crossing * ew.astype(np.uint64)).sum(dtype=np.uint64)) // 2
    loads = np.zeros(k, np.uint64)
    np.add.at(loads, labels, np.uint64(1) if vw is None else vw.astype(np.uint64))
    dev = [None if a is None else torch.from_numpy(a.view(np.int32)).cuda() for a in (off, nbr, vw, ew, labels)]
    ptr = [None if t is None else t.data_ptr() for t in dev]
    stream = torch.cuda.current_stream().cuda_stream
    for call in (ctx.evaluate_device, gp.evaluate_device_static):
        out = torch.full((k + 1,), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        call(ptr[0], ptr[1], n, m, ptr[2], ptr[3], ptr[4], k, out.data_ptr(), out.data_ptr() + 8, stream)
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(np.uint64)
        assert int(got[0]) == cut
        assert (got[1:] == loads).all()


@pytest.mark.parametrize("where", [0, 255, 256, 4095, -1])
def test_one_wrong_neighbour_is_counted_once(gp, ctx, where):
    import torch
    n, deg = 3000, 5
    off = np.arange(n + 1, dtype=np.int32) * deg
    nbr = np.zeros(n * deg, np.int32)
    nbr[where] = n
    dev = [torch.from_numpy(a).cuda() for a in (off, nbr, np.zeros(n, np.int32))]
    out = torch.zeros(3, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(gp.GpartError, match="^GP_INVALID_ARGUMENT: 1 labels"):
        ctx.evaluate_device(dev[0].data_ptr(), dev[1].data_ptr(), n, n * deg, None, None, dev[2].data_ptr(), 2,
                            out.data_ptr(), out.data_ptr() + 8)
