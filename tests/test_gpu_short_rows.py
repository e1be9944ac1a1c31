"""Rows of at most 32 entries against the oracle: two contraction rows per warp
(both at most 16 entries, or one longer), and movers of at most 8 entries that
one thread decides, with self-loops, repeated neighbours and zero weights."""
import numpy as np
import pytest

import horkxg_b200 as hb
import pyoracle as O

pytestmark = pytest.mark.gpu


def rows_graph(lengths, n_targets, seed, max_w):
    rng = np.random.default_rng(seed)
    rows = len(lengths)
    off = np.zeros(rows + n_targets + 1, np.int64)
    off[1:rows + 1] = np.cumsum(lengths)
    off[rows + 1:] = off[rows]
    nbr = rows + rng.integers(0, n_targets, off[rows])
    return off, nbr, rng.integers(1, max_w, off[rows]).astype(np.uint64), rows + n_targets


@pytest.mark.parametrize("width,scale", [(hb.STANDARD, 1), (hb.BIG, 1 << 40)])
@pytest.mark.parametrize("lengths", [[16] * 8, [1, 16, 17, 2, 16, 32, 32, 32, 5], [32] * 3, [1], [0, 3, 0, 31, 15]])
@pytest.mark.parametrize("targets", [3, 20, 5000])
def test_contract_short_rows(ctx, width, scale, lengths, targets):
    off, nbr, ew, n = rows_graph(lengths, targets, 7, 100)
    ew = ew * np.uint64(scale)
    mapping = np.arange(n, dtype=np.int32)
    mapping[-1] = n - 2   # one merged pair of targets
    coarse = int(mapping.max()) + 1
    coff, cnbr, cew, cvw = ctx.contract(hb.HostGraph(off, nbr, ew, width=width, index64=True), mapping, coarse)
    want = O.contract(O.Graph(off, nbr, ew), mapping, coarse)
    assert np.array_equal(coff, want.off) and np.array_equal(cnbr, want.nbr)
    assert np.array_equal(cew, want.ew) and np.array_equal(cvw, want.vw)


@pytest.mark.parametrize("width,scale", [(hb.STANDARD, 1), (hb.BIG, 1 << 40)])
@pytest.mark.parametrize("max_degree", [1, 8, 9, 32])
def test_short_movers(ctx, width, scale, max_degree):
    rng = np.random.default_rng(max_degree)
    n = 3001
    off = np.concatenate([[0], np.cumsum(rng.integers(0, max_degree + 1, n))]).astype(np.int64)
    row = np.repeat(np.arange(n), np.diff(off))
    nbr = np.where(rng.random(len(row)) < 0.1, row, (row + rng.integers(-4, 5, len(row))) % n)
    order = np.lexsort((nbr, row))
    nbr = nbr[order]
    ew = (rng.integers(0, 4, len(nbr)) * scale).astype(np.uint64)
    vw = rng.integers(0, 5, n).astype(np.uint64)
    for level, beta, pack in ((0, 16, False), (1, 2, False)):
        mp, cn, cap = ctx.aggregate(hb.HostGraph(off, nbr, ew, vw, width=width, index64=True), 4, 3, level, beta, pack)
        omp, ocn, ocap = O.aggregate(O.Graph(off, nbr, ew, vw), 4, 3, level, beta, pack)
        assert (cn, cap) == (ocn, ocap) and np.array_equal(mp, omp)
