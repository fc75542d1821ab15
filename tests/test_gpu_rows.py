"""Pulls over the hot-source rows (32-vertex slices of column-major lists) at
the sizes where slices, columns and chunks end: vertex counts around a slice,
list lengths around the four-entry columns, the light bound and a chunk, and
vertices without in-edges between them; against the oracle."""
import numpy as np
import pytest

import geminigraph_gb300 as gg
from oracle.oracle import OracleGraph

pytestmark = pytest.mark.gpu


def lists_graph(V, lengths, seed):
    """dst i has lengths[i % len(lengths)] in-edges from random sources."""
    rng = np.random.default_rng(seed)
    deg = np.resize(np.asarray(lengths, np.int64), V)
    dst = np.repeat(np.arange(V, dtype=np.uint32), deg)
    src = rng.integers(0, V, len(dst)).astype(np.uint32)
    return src, dst, rng.random(len(dst), dtype=np.float32)


def rel_l1(a, b):
    return float(np.abs(a - b).sum() / max(np.abs(b).sum(), 1e-300))


@pytest.mark.parametrize("V", [1, 31, 32, 33, 257, 1000])
@pytest.mark.parametrize("lengths", [[0], [1], [3, 4, 5, 0], [7, 8, 9], [31, 32, 33, 0, 1], [511, 512, 513, 2, 0],
                                     [1500, 0, 1]])
@pytest.mark.parametrize("light,chunk", [(0, 0), (1, 128), (8, 512), (1024, 256)])
def test_rows_match_oracle(V, lengths, light, chunk):
    s, d, w = lists_graph(V, lengths, V + len(lengths))
    g = gg.Graph.from_edges(V, s, d, w)
    gs = gg.Graph.from_edges(V, s, d, symmetric=True)
    if light:
        g.set_bins(light, chunk)
        gs.set_bins(light, chunk)
    o = OracleGraph(V, s, d, w)
    for n in (1, 2, 3, 6):
        oranks, _, otr = o.pagerank(n)
        ranks, _, st = g.pagerank(n)
        assert rel_l1(ranks, oranks) < 1e-10 and st.rows() == otr
        r32, _, _ = g.pagerank(n, f32=True)
        assert rel_l1(r32.astype(np.float64), oranks) < 1e-5
    root = int(s[0]) if len(s) else 0
    odist, otr = o.sssp(root)
    dist, st = g.sssp(root)
    assert np.array_equal(dist.view(np.uint32), odist.view(np.uint32)) and st.rows() == otr
    odep, oinv, otr = o.bc(root)
    dep, inv, st = g.bc(root)
    assert np.array_equal(np.isnan(dep), np.isnan(odep)) and np.array_equal(inv, oinv) and st.rows() == otr
    ok = ~np.isnan(odep)
    assert rel_l1(dep[ok], odep[ok]) < 1e-10
    olabel, otr = OracleGraph(V, s, d, symmetric=True).cc()
    label, st = gs.cc()
    assert np.array_equal(label, olabel) and st.rows() == otr
    g.close()
    gs.close()


def test_float_delta_of_large_degrees():
    """The float deltas of sources with more out-edges than a float counts (2^24)."""
    V, hub = 64, (1 << 24) + 3
    s = np.zeros(hub + V, np.uint32)
    d = (np.arange(hub + V, dtype=np.uint32) * 7 + 1) % V
    s[hub:] = np.arange(V)
    g = gg.Graph.from_edges(V, s, d)
    _, d64, _ = g.pagerank(4)
    _, d32, _ = g.pagerank(4, f32=True)
    assert np.allclose(d32, d64, rtol=1e-5, atol=1e-6)
