"""Whole traversals on the device (cooperative launches): values bit-identical
to the oracle's and the same per-call trace at the sizes where the runs'
pieces end: one vertex, a queue of only hubs, lists around the hub bound (128)
and the heavy bound (2048), more calls than one launch records (1536),
vertices without out-edges in the frontier, and sparse, dense and mixed
calls; a second run and a run of another root reuse the buffers."""
import numpy as np
import pytest

import geminigraph_gb300 as gg
from oracle.oracle import OracleGraph, bfs_levels

pytestmark = pytest.mark.gpu


def chain(n):
    s = np.arange(n - 1, dtype=np.uint32)
    return n, s, s + 1


def hubs(V, lengths):
    """Vertices 0.. with out-lists (and mirrored in-lists) of the given lengths, joined in a ring."""
    rng = np.random.default_rng(V)
    s, d = [np.arange(len(lengths))], [(np.arange(len(lengths)) + 1) % len(lengths)]
    for i, n in enumerate(lengths):
        t = rng.integers(0, V, n)
        s += [np.full(n, i), t[::2]]
        d += [t, np.full(len(t[::2]), i)]
    return V, np.concatenate(s).astype(np.uint32), np.concatenate(d).astype(np.uint32)


def rmat(scale, ef):
    r = gg.generate_records(gg.RMAT, scale, ef, 7).view(np.uint32).reshape(-1, 2)
    return 1 << scale, r[:, 0].copy(), r[:, 1].copy()


GRAPHS = {
    "single": (1, np.zeros(2, np.uint32), np.zeros(2, np.uint32)),
    "empty": (70, np.zeros(0, np.uint32), np.zeros(0, np.uint32)),
    "chain": chain(1700),
    "long-chain": chain(3300),
    "hubs": hubs(4000, [127, 128, 129, 1, 2047, 2048, 2049, 600]),
    "only-hubs": hubs(300, [500, 400, 300]),
    "star": (9000, np.zeros(8999, np.uint32), np.arange(1, 9000, dtype=np.uint32)),
    "rmat9": rmat(9, 16),
    "rmat13": rmat(13, 3),
    "rmat15": rmat(15, 24),
}


@pytest.mark.parametrize("layout", [True, False])
@pytest.mark.parametrize("name", GRAPHS)
def test_traversals(name, layout):
    """layout False: no rows to pull, so CC and SSSP enter the device for
    their runs of small sparse calls only, from the host loop and back."""
    V, s, d = GRAPHS[name]
    rng = np.random.default_rng(len(s))
    w = rng.random(len(s), dtype=np.float32)
    g = gg.Graph.from_edges(V, s, d, w)
    gs = gg.Graph.from_edges(V, s, d, w, symmetric=True)
    g.set_pr_layout(layout)
    gs.set_pr_layout(layout)
    o, os_ = OracleGraph(V, s, d, w), OracleGraph(V, s, d, w, symmetric=True)
    olabel, octr = os_.cc()
    for root in sorted({0, V - 1, V // 3}):
        for gr, orc in ((g, o), (gs, os_)):
            odist, otr = orc.sssp(root)
            dist, st = gr.sssp(root)
            assert np.array_equal(dist.view(np.uint32), odist.view(np.uint32))
            assert st.rows() == otr
            oparent, otr = orc.bfs(root)
            parent, st = gr.bfs(root)
            assert np.array_equal(bfs_levels(parent, root), bfs_levels(oparent, root))
            assert st.rows() == otr
        label, st = gs.cc()
        assert np.array_equal(label, olabel) and st.rows() == octr
    g.close()
    gs.close()
