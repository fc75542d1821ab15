"""BC of one root at the sizes where its level and renumbering kernels can go
wrong: bitmaps' word edges, no edges (every call dense, levels empty), vertices
that are not reached (inverse path counts infinite, dependencies NaN), deep
chains, a second call on the same workspaces; against the oracle.  Path counts
are whole numbers, so their inverses are equal; dependencies are sums in
another order: relative L1 within 1e-10, as everywhere in these tests."""
import numpy as np
import pytest

import geminigraph_gb300 as gg
from oracle.oracle import OracleGraph

pytestmark = pytest.mark.gpu


def edges(V, shape, rng):
    if shape == "none":
        return np.zeros(0, np.uint32), np.zeros(0, np.uint32)
    if shape == "chain":  # the upper half of the chain is not reached from its middle
        return np.arange(V - 1, dtype=np.uint32), np.arange(1, V, dtype=np.uint32)
    n = 6 * V
    half = max(1, V // 2)  # sources in the lower half only, skewed
    return ((half * rng.random(n) ** 3).astype(np.uint32), rng.integers(0, V, n).astype(np.uint32))


@pytest.mark.parametrize("layout", [True, False])
@pytest.mark.parametrize("V,shape", [(1, "none"), (33, "none"), (32, "skewed"), (33, "skewed"), (97, "chain"),
                                     (1025, "skewed"), (40001, "skewed")])
def test_one_root(V, shape, layout):
    s, d = edges(V, shape, np.random.default_rng(V))
    g = gg.Graph.from_edges(V, s, d)
    g.set_pr_layout(layout)
    o = OracleGraph(V, s, d)
    for root in sorted({0, V // 3, V - 1}):
        dep, inv, st = g.bc(root)
        odep, oinv, otr = o.bc(root)
        assert np.array_equal(inv, oinv)
        assert np.array_equal(np.isnan(dep), np.isnan(odep))
        ok = ~np.isnan(odep)
        assert np.abs(dep[ok] - odep[ok]).sum() <= 1e-10 * max(np.abs(odep[ok]).sum(), 1e-300)
        assert [r[:2] for r in st.rows()] == [r[:2] for r in otr]
    g.close()
