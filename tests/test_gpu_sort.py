"""The build's radix sort at the edges of its tiles (6144 entries), of its
digits (vertex counts around powers of two, so 1 to 6 passes of unequal
width) and with duplicate edges, whose weights must keep the records' order
in both directions: against numpy's stable sort."""
import numpy as np
import pytest

import geminigraph_gb300 as gg

pytestmark = pytest.mark.gpu


def side(major, minor, w, V):
    order = np.lexsort((np.arange(len(major)), minor, major))
    off = np.zeros(V + 1, np.uint64)
    np.cumsum(np.bincount(major, minlength=V), out=off[1:])
    return off, minor[order], w[order]


@pytest.mark.parametrize("V", [1, 2, 3, 255, 257, 4096, 65537, 1 << 20])
@pytest.mark.parametrize("E", [0, 1, 2, 6143, 6144, 6145, 50000])
@pytest.mark.parametrize("symmetric", [False, True])
def test_adjacency_equals_stable_sort(V, E, symmetric):
    rng = np.random.default_rng(V * 7 + E)
    # a few hubs and many duplicates
    src = np.minimum(rng.integers(0, V, E), rng.integers(0, V, E)).astype(np.uint32)
    dst = (rng.integers(0, V, E) // np.uint32(1 + E % 3)).astype(np.uint32)
    w = rng.random(E, dtype=np.float32)
    g = gg.Graph.from_edges(V, src, dst, w, symmetric=symmetric)
    s, d, ww = (np.concatenate([src, dst]), np.concatenate([dst, src]), np.concatenate([w, w])) if symmetric \
        else (src, dst, w)
    for incoming in (False, True):
        a, b = (d, s) if incoming and not symmetric else (s, d)
        off, nbr, wt, deg = g.adjacency(incoming)
        eoff, enbr, ewt = side(a, b, ww, V)
        assert np.array_equal(off, eoff)
        assert np.array_equal(nbr, enbr)
        assert np.array_equal(wt.view(np.uint32), ewt.view(np.uint32))
        assert np.array_equal(deg, np.diff(eoff).astype(np.uint32))


@pytest.mark.parametrize("V", [3, 1000, 70000])
def test_layout_keeps_results(V):
    """Toolkits on the hot-source layout (built by the same sort) against the plain adjacency."""
    rng = np.random.default_rng(V)
    E = 9 * V + 5
    src, dst = (np.minimum(rng.integers(0, V, E), rng.integers(0, V, E)).astype(np.uint32) for _ in range(2))
    w = rng.random(E, dtype=np.float32)
    a, b = (gg.Graph.from_edges(V, src, dst, w) for _ in range(2))
    b.set_pr_layout(False)
    root = int(src[0])
    assert np.array_equal(a.sssp(root)[0], b.sssp(root)[0])
    ra, rb = a.pagerank(5)[0], b.pagerank(5)[0]
    assert np.abs(ra - rb).sum() <= 1e-13 * np.abs(rb).sum()
    (da, ia, _), (db, ib, _) = a.bc(root), b.bc(root)
    assert np.array_equal(ia, ib)
    ok = np.isfinite(db)
    assert np.array_equal(np.isnan(da), np.isnan(db))
    assert np.abs(da[ok] - db[ok]).sum() <= 1e-10 * max(np.abs(db[ok]).sum(), 1e-300)
