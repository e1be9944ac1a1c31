"""The rebalance's selection inside the bucket that crosses a part's quota
(src/refine_incremental.cuh:188-232), against the oracle's sorted ranks: lists
of every size class of the threshold search (ranked directly, staged in
shared memory, read from global memory), with equal and with distinct gains
and weights."""
import numpy as np
import pytest

import horkxg_b200 as hb
import pyoracle as O

pytestmark = pytest.mark.gpu


def pairs_graph(pairs, k, weighted, seed):
    """Disjoint edges whose ends lie in different parts, so that the LP round
    pulls one end of each across and overloads parts by many vertices of
    equal (unit) or varied (weighted) gain; a path keeps gains apart."""
    rng = np.random.default_rng(seed)
    n = 2 * pairs
    a = np.arange(0, n, 2)
    b = a + 1
    w = rng.integers(1, 50, pairs) if weighted else np.ones(pairs, np.int64)
    src, dst, ew = np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w])
    if weighted:
        p = np.arange(n - 2)
        pw = rng.integers(1, 9, n - 2)
        src, dst, ew = (np.concatenate(x) for x in ((src, p, p + 2), (dst, p + 2, p), (ew, pw, pw)))
    order = np.lexsort((dst, src))
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=n), out=off[1:])
    vw = rng.integers(1, 4, n).astype(np.uint64) if weighted else None
    # part 0 holds nothing but larger ends; the smaller end of a cut pair
    # moves, so the first round doubles part 0; the other pairs are internal
    labels = np.empty(n, np.int32)
    cut = 2 * pairs // k
    labels[a[:cut]] = 1 + np.arange(cut) % (k - 1)
    labels[b[:cut]] = 0
    labels[a[cut:]] = labels[b[cut:]] = 1 + np.arange(pairs - cut) % (k - 1)
    return off, dst[order], ew[order].astype(np.uint64) if weighted else None, vw, labels


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("pairs,k", [(40, 2), (700, 2), (2100, 3), (17000, 2), (60000, 2), (50000, 5)])
def test_rebalance_selection_matches_oracle(ctx, pairs, k, weighted):
    off, nbr, ew, vw, labels = pairs_graph(pairs, k, weighted, pairs + k)
    ratio = 1.03
    total = int(vw.sum()) if weighted else len(labels)
    loads = np.bincount(labels, weights=None if vw is None else vw.astype(float), minlength=k)
    while loads.max() > hb.capacity(total, k, ratio):   # the start has to be balanced
        ratio += 0.05
    g = hb.HostGraph(off, nbr, ew, vw, index64=True)
    og = O.Graph(off, nbr, ew, vw)
    olab, ost = O.refine(og, labels, k, ratio, 8)
    assert ost.admission_iterations > 0
    for det in (True, False):   # the default mode ranks as the deterministic one does
        lab, st = ctx.refine(g, labels, k, ratio, 8, det)
        assert np.array_equal(lab, olab)
        assert (st.rounds, st.final_cut, st.admission_iterations) == (ost.rounds, ost.final_cut, ost.admission_iterations)
