"""CC's floor (the least vertex with an out-edge): labels and the per-call
trace where the large component does not hold it, where it lies past the first
bitmap words, on several components and without edges; against the oracle."""
import numpy as np
import pytest

import geminigraph_gb300 as gg
from oracle.oracle import OracleGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [True, False])
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("V,first,parts", [(1, 0, 1), (64, 0, 1), (5000, 40, 3), (70000, 33000, 2), (70000, 0, 500)])
def test_components(V, first, parts, symmetric, layout):
    rng = np.random.default_rng(V + first + parts)
    # parts interleaved components over [first, V), component 0 a single pair where there are others
    ids = np.arange(first, V, dtype=np.int64)
    s, d = [], []
    for p in range(parts):
        own = ids[p::parts][:2] if p == 0 and parts > 1 else ids[p::parts]
        if len(own) < 2:
            continue
        n = 3 * len(own)
        s.append(own[np.minimum(rng.integers(0, len(own), n), rng.integers(0, len(own), n))])
        d.append(own[rng.integers(0, len(own), n)])
    s = np.concatenate(s).astype(np.uint32) if s else np.zeros(0, np.uint32)
    d = np.concatenate(d).astype(np.uint32) if d else np.zeros(0, np.uint32)
    g = gg.Graph.from_edges(V, s, d, symmetric=symmetric)
    g.set_pr_layout(layout)
    olabel, otr = OracleGraph(V, s, d, symmetric=symmetric).cc()
    for _ in range(2):
        label, st = g.cc()
        assert np.array_equal(label, olabel)
        assert st.rows() == otr
    g.close()
