"""Contraction rows sorted in shared memory by buckets, against the oracle:
even keys, keys crowded into one bucket (equal, and distinct so that a warp or
the radix sort has to order them), rows of sentinels only, at the class bounds
257, 1,024 and 4,096."""
import numpy as np
import pytest

import horkxg_b200 as hb
import pyoracle as O

pytestmark = pytest.mark.gpu


def fan(lengths, spread, n_targets, seed):
    """Row i (a coarse vertex of its own) gets lengths[i] entries whose targets
    come from spread[i](rng, length); targets are further coarse vertices."""
    rng = np.random.default_rng(seed)
    rows = len(lengths)
    n = rows + n_targets
    off = np.zeros(n + 1, np.int64)
    nbr = []
    for i, (l, f) in enumerate(zip(lengths, spread)):
        t = f(rng, l)
        nbr.append(np.where(t < 0, i, rows + t))
        off[i + 1] = off[i] + l
    off[rows + 1:] = off[rows]
    return off, np.concatenate(nbr), n


def even(n):
    return lambda rng, l: rng.integers(0, n, l)


def crowd(n, share, width):
    """Most targets within `width` ids of one place, the rest anywhere."""
    def f(rng, l):
        t = rng.integers(0, n, l)
        near = rng.random(l) < share
        t[near] = n // 3 + rng.integers(0, width, near.sum())
        return t
    return f


def internal(rng, l):
    return np.full(l, -1)


@pytest.mark.parametrize("width,scale", [(hb.STANDARD, 1), (hb.BIG, 1 << 40)])
def test_bucket_rows_match_oracle(ctx, width, scale):
    n = 400_000   # coarse_n / 64 is above 4,096: rows are not ranked by the bitmap
    lengths, spread = [], []
    for l in (257, 258, 700, 1024, 1025, 2048, 3000, 4095, 4096):
        for f in (even(n), even(40), crowd(n, 0.5, 1), crowd(n, 0.03, 1), crowd(n, 0.2, 30), crowd(n, 0.9, 900),
                  crowd(n, 1.0, 5), internal):
            lengths.append(l)
            spread.append(f)
    off, nbr, total = fan(lengths, spread, n, 3)
    ew = (np.random.default_rng(4).integers(1, 1000, len(nbr)) * scale).astype(np.uint64)
    mapping = np.arange(total, dtype=np.int32)
    coff, cnbr, cew, cvw = ctx.contract(hb.HostGraph(off, nbr, ew, width=width, index64=True), mapping, total)
    o = O.contract(O.Graph(off, nbr, ew), mapping, total)
    assert np.array_equal(coff, o.off) and np.array_equal(cnbr, o.nbr) and np.array_equal(cew, o.ew)
