"""The build's two sorts share digit counts: those of the first are taken while
the keys are made, and the second starts from the first's places where their
digits agree.  Both directions at every kind of width (one to four digits per
id, digits that do and do not span both ids), tiny and ragged record counts,
against numpy's stable sort."""
import numpy as np
import pytest

import geminigraph_gb300 as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 4, 5, 7, 8, 9, 12, 13, 14, 15, 16, 17, 20, 21, 22, 23, 24])
@pytest.mark.parametrize("E", [1, 2, 511, 20011])
def test_both_directions(bits, E):
    V = (1 << bits) - (bits > 1)
    rng = np.random.default_rng(bits * 31 + E)
    src = (V * rng.random(E) ** 2).astype(np.uint32)
    dst = rng.integers(0, V, E).astype(np.uint32)
    dst[: E // 3] = V - 1
    w = rng.random(E, dtype=np.float32)
    g = gg.Graph.from_edges(V, src, dst, w)
    for incoming in (False, True):
        major, minor = (dst, src) if incoming else (src, dst)
        order = np.lexsort((np.arange(E), minor, major))
        off, nbr, wt, _ = g.adjacency(incoming)
        eoff = np.zeros(V + 1, np.uint64)
        np.cumsum(np.bincount(major, minlength=V), out=eoff[1:])
        assert np.array_equal(off, eoff)
        assert np.array_equal(nbr, minor[order])
        assert np.array_equal(wt.view(np.uint32), w[order].view(np.uint32))
    g.close()
