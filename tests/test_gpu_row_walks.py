"""Kernels that walk rows in groups -- the cut, the part weights, the analyzer,
the neighbour check and the hub index -- on row lengths around their group
sizes (0, 8, 32, 33, the hub degree 2,048 and above), on arrays that start at
any entry, and on weights above 2^26."""
import ctypes

import numpy as np
import pytest
import torch

import horkxg_b200 as hb

pytestmark = pytest.mark.gpu


def rows_graph(lengths, n, seed):
    """Directed rows of the given lengths (the recount does not need symmetry)."""
    rng = np.random.default_rng(seed)
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(lengths)
    return off, rng.integers(0, n, off[-1])


LENGTHS = [0, 1, 7, 8, 9, 31, 32, 33, 64, 255, 2047, 2048, 2049, 4097, 9000]


@pytest.mark.parametrize("n", [1, 3, 45, 1001])
@pytest.mark.parametrize("width,scale", [(hb.STANDARD, 0), (hb.STANDARD, 1), (hb.STANDARD, 1 << 25), (hb.BIG, 1 << 40)])
def test_cut_loads_and_analysis_match_numpy(ctx, n, width, scale):
    rng = np.random.default_rng(n)
    lengths = np.array([LENGTHS[i % len(LENGTHS)] if n <= 45 or i % 29 == 0 else i % 12 for i in range(n)])
    off, nbr = rows_graph(lengths, n, n)
    ew = vw = None
    if scale:
        ew = rng.integers(1, 60, len(nbr)).astype(np.uint64) * scale
        vw = rng.integers(1, 60, n).astype(np.uint64) * scale
    k = min(7, max(2, n))
    labels = rng.integers(0, k, n).astype(np.int32)
    g = hb.HostGraph(off, nbr, ew, vw, width=width, index64=True)
    cut, loads = ctx.cut(g, labels, k)
    src = np.repeat(labels, np.diff(off))
    dst = labels[nbr]
    w = np.ones(len(nbr), np.uint64) if ew is None else ew
    v = np.ones(n, np.uint64) if vw is None else vw
    cross = src != dst
    assert cut == int(w[cross].sum())
    assert list(loads) == [int(v[labels == p].sum()) for p in range(k)]
    per, summary = ctx.analyze(g, labels, k)
    for p in range(k):
        assert per["vertices"][p] == (labels == p).sum()
        assert per["weighted_internal"][p] == int(w[~cross & (src == p)].sum())
        assert per["weighted_outgoing"][p] == int(w[cross & (src == p)].sum())
        assert per["weighted_incoming"][p] == int(w[cross & (dst == p)].sum())
        assert per["internal_edges"][p] == (~cross & (src == p)).sum()
        assert per["incoming_cut_edges"][p] == (cross & (dst == p)).sum()
    assert summary["directed_edge_cut"] == cross.sum()


@pytest.mark.parametrize("parts", [1, 257, 1024])
def test_analysis_of_many_parts(ctx, parts):
    off, nbr = rows_graph(np.full(3000, 9), 3000, 1)
    labels = (np.arange(3000) % parts).astype(np.int32)
    per, _ = ctx.analyze(hb.HostGraph(off, nbr, index64=True), labels, parts)
    src = np.repeat(labels, 9)
    assert np.array_equal(per["outgoing_cut_edges"], np.bincount(src[src != labels[nbr]], minlength=parts))


@pytest.mark.parametrize("start", [0, 1, 2, 3])
@pytest.mark.parametrize("m", [0, 1, 2, 3, 4, 5, 9, 70001])
def test_neighbor_check_at_any_alignment(ctx, start, m):
    """Every entry is checked once, whatever the array's first address; the
    array is passed in place."""
    n = 50
    off = torch.full((n + 1,), m, dtype=torch.int32, device="cuda")
    off[0] = 0
    room = torch.full((m + 8,), -7, dtype=torch.int32, device="cuda")   # around the array: never read
    nbr = room[start:start + m]
    nbr.copy_(torch.arange(m, device="cuda", dtype=torch.int32) % n)
    labels = torch.zeros(n, dtype=torch.int32, device="cuda")

    def analyze():
        torch.cuda.synchronize()
        d = hb.GraphDesc()
        d.n, d.m, d.width, d.memory, d.index64 = n, m, hb.STANDARD, hb.DEVICE, 0
        d.offsets, d.neighbors = off.data_ptr(), nbr.data_ptr()
        return hb.lib().gp_analyze(ctx._h, ctypes.byref(d), labels.data_ptr(), 1, None, None)

    assert analyze() == 0
    for at in sorted({0, m // 2, m - 1}):
        if 0 <= at < m:
            for bad in (-1, n):
                keep = int(nbr[at])
                nbr[at] = bad
                assert analyze() == hb.GP_ERUNTIME
                nbr[at] = keep
    assert analyze() == 0


def test_labels_out_of_range_are_rejected(ctx):
    off, nbr = rows_graph(np.full(10, 2), 10, 0)
    g = hb.HostGraph(off, nbr, index64=True)
    for bad in (-1, 3):
        labels = np.zeros(10, np.int32)
        labels[9] = bad
        for call in (lambda: ctx.cut(g, labels, 3), lambda: ctx.refine(g, labels, 3)):
            with pytest.raises(hb.PartitionError) as e:
                call()
            assert e.value.status == hb.GP_EINVAL
