"""The diffusion with replicated vectors (cluster and grid forms) against the
general kernel, bit for bit, and the fused sort and split against the oracle's
replay, at the sizes where the forms change: rows of 32 and 33 entries and
around 128 (unit weights take another rounding in the last partial block),
4,096 and 8,192 positions, 2^18 entries."""
import numpy as np
import pytest

import horkxg_b200 as hb
import pyoracle as O
from horkxg_b200 import graphs
from test_gpu_parity import dense_random_csr

pytestmark = pytest.mark.gpu


def circulant(n, degree):
    """Every row has exactly `degree` entries (degree even)."""
    steps = np.concatenate([np.arange(1, degree // 2 + 1), n - np.arange(1, degree // 2 + 1)])
    nbr = np.sort((np.arange(n)[:, None] + steps[None, :]) % n, axis=1)
    return np.arange(n + 1, dtype=np.int64) * degree, nbr.reshape(-1)


def weights(off, nbr):
    src = np.repeat(np.arange(len(off) - 1), np.diff(off))
    a, b = np.minimum(src, nbr), np.maximum(src, nbr)
    return ((a * 2654435761 + b * 40503) % 97 + 1).astype(np.uint64)


CASES = [("rgg", 33, 10), ("rgg", 1023, 10), ("rgg", 1025, 10), ("rgg", 4096, 10), ("rgg", 4097, 10), ("rgg", 8192, 10),
         ("rgg", 8193, 10), ("circulant", 900, 32), ("circulant", 900, 34), ("circulant", 900, 128),
         ("circulant", 900, 130), ("circulant", 900, 290), ("circulant", 900, 292), ("dense", 1500, 200)]


def make(kind, n, degree):
    if kind == "rgg":
        return graphs.rgg_csr(n, float(degree), n)
    return circulant(n, degree) if kind == "circulant" else dense_random_csr(n, degree, 3)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("kind,n,degree", CASES)
def test_fast_diffusion_equals_general(ctx, kind, n, degree, weighted):
    off, nbr = make(kind, n, degree)
    g = hb.HostGraph(off, nbr, weights(off, nbr) if weighted else None)
    k = 2 if n < 100 else 8
    with hb.Context(0) as general:
        general.set_small_diffusion(False)
        for seed in (0, 5):
            la, ta = ctx.initial_partition_trace(g, k, 1.05, seed)
            lb, tb = general.initial_partition_trace(g, k, 1.05, seed)
            assert np.array_equal(ta.view(np.uint32), tb.view(np.uint32))
            assert np.array_equal(la, lb)
            olab, err = O.initial_partition_replay(O.Graph(off, nbr, g.ew), k, ta, 1.05, seed)
            assert np.array_equal(la, olab) and err <= 1e-5


def test_fast_diffusion_rows_without_group_edges(ctx):
    """Vertices whose neighbours all lie outside the group keep their value."""
    off, nbr = circulant(600, 40)
    labels = (np.arange(600) % 2).astype(np.int32)
    labels[::50] = 7
    g = hb.HostGraph(off, nbr)
    with hb.Context(0) as general:
        general.set_small_diffusion(False)
        for group in (0, 7):
            a, b = ctx.diffusion(g, labels, group, 1, 64), general.diffusion(g, labels, group, 1, 64)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
