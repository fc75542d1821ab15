"""SSSP's weight-ordered lists (walks end where the least active distance plus
the next weight reaches the vertex's own): distances bit-identical to the
oracle's and the per-call trace equal, for weights whose range, sign and
repetition put class bounds in awkward places, pulling every dense call."""
import numpy as np
import pytest

import geminigraph_gb300 as gg
import graphgen
from oracle.oracle import OracleGraph

pytestmark = pytest.mark.gpu


def weights(kind, n, rng):
    u = rng.random(n, dtype=np.float32)
    return {
        "unit": u,
        "equal": np.full(n, 0.25, np.float32),
        "zero": np.zeros(n, np.float32),
        "offset": (u + np.float32(1000)).astype(np.float32),
        "wide": (u.astype(np.float64) ** 12 * 1e6).astype(np.float32),
        "tiny": (u * np.float32(1e-30)).astype(np.float32),
        "integers": rng.integers(1, 200, n).astype(np.float32),
        "huge": np.where(u < 0.01, np.float32(3e38), u).astype(np.float32),
        "infinite": np.where(u < 0.01, np.float32(np.inf), u).astype(np.float32),
    }[kind]


@pytest.mark.parametrize("kind", ["unit", "equal", "zero", "offset", "wide", "tiny", "integers", "huge", "infinite"])
@pytest.mark.parametrize("V", [33, 4096, 30000])
@pytest.mark.parametrize("symmetric", [False, True])
def test_distances(kind, V, symmetric):
    rng = np.random.default_rng(V)
    if V == 4096:
        s, d, _ = graphgen.rmat(12, 16, 5, weighted=True)
    else:
        s, d = (np.minimum(rng.integers(0, V, 20 * V), rng.integers(0, V, 20 * V)).astype(np.uint32) for _ in range(2))
    w = weights(kind, len(s), rng)
    g = gg.Graph.from_edges(V, s, d, w, symmetric=symmetric)
    o = OracleGraph(V, s, d, w, symmetric=symmetric)
    for root in {int(s[0]), int(d[1]), V - 1}:
        odist, otr = o.sssp(root)
        for div in (None, 0, 4):
            if div is not None:
                g.set_dense_push(div)
            dist, st = g.sssp(root)
            assert np.array_equal(dist.view(np.uint32), odist.view(np.uint32))
            assert st.rows() == otr
    g.close()
