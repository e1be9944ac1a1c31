"""Symmetrising row by row against the numpy restatement of the reference's
tool: rows of every size class, duplicates and self loops, host and device
arrays, both neighbour widths, the capacity check, and a graph just above the
row form's vertex bound."""
import ctypes

import numpy as np
import pytest
import torch

import horkxg_b200 as hb
import pyoracle as O

pytestmark = pytest.mark.gpu


def directed(n, m, hubs, seed):
    """Random entries, some duplicated and some self loops, with `hubs` popular
    targets drawing a third of them."""
    rng = np.random.default_rng(seed)
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    if m:
        dst[: m // 3] = rng.integers(0, hubs, m // 3)
        dst[m // 2: m // 2 + m // 20] = src[m // 2: m // 2 + m // 20]
        src[-(m // 10) - 1:], dst[-(m // 10) - 1:] = src[: m // 10 + 1], dst[: m // 10 + 1]
    order = np.argsort(src, kind="stable")
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=n), out=off[1:])
    return off, dst[order]


CASES = [(1, 0, 1), (1, 5, 1), (2, 3, 1), (40, 200, 2), (3000, 20, 3), (5000, 40000, 5), (70000, 500000, 40),
         (70000, 500000, 1), (200000, 300000, 1), (4_200_000, 50000, 3)]


@pytest.mark.parametrize("n,m,hubs", CASES)
@pytest.mark.parametrize("bytes_", [8, 4])
def test_symmetrize_rows_match_numpy(ctx, n, m, hubs, bytes_):
    off, nbr = directed(n, m, hubs, n + m)
    want_off, want_nbr, loops = O.symmetrize(off, nbr)[:3]
    got_off, got_nbr, info = ctx.symmetrize(hb.HostGraph(off, nbr, index64=True), neighbor_bytes=bytes_)
    assert np.array_equal(got_off, want_off) and np.array_equal(got_nbr, want_nbr)
    assert info.output_directed_edges == len(want_nbr) == 2 * info.unique_undirected_edges
    src = np.repeat(np.arange(n), np.diff(off))
    assert info.self_loops_removed == int((src == nbr).sum())


def test_symmetrize_rows_on_device_and_capacity(ctx):
    off, nbr = directed(3000, 30000, 4, 9)
    want_off, want_nbr = O.symmetrize(off, nbr)[:2]
    dev = [torch.from_numpy(x.astype(np.int32)).cuda() for x in (off, nbr)]
    out_off = torch.full((3001,), -5, dtype=torch.int64, device="cuda")
    out_nbr = torch.full((60000,), -5, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    d = hb.GraphDesc()
    d.n, d.m, d.width, d.memory, d.index64 = 3000, 30000, hb.STANDARD, hb.DEVICE, 0
    d.offsets, d.neighbors = dev[0].data_ptr(), dev[1].data_ptr()
    info = hb.SymmetrizeInfo()

    def call(capacity):
        return hb.lib().gp_symmetrize(ctx._h, ctypes.byref(d), out_off.data_ptr(), out_nbr.data_ptr(), 8, capacity,
                                      ctypes.byref(info))

    assert call(len(want_nbr) - 1) == hb.GP_EINVAL
    assert info.output_directed_edges == len(want_nbr)
    assert int(out_off.min()) == int(out_off.max()) == -5 and int(out_nbr.max()) == -5   # nothing written
    assert call(len(want_nbr)) == 0
    assert np.array_equal(out_off.cpu().numpy(), want_off)
    assert np.array_equal(out_nbr[:len(want_nbr)].cpu().numpy(), want_nbr)
    assert int(out_nbr[len(want_nbr):].max()) == -5
