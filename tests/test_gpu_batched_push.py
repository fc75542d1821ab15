"""The batched relaxation where its tiles and runs can go wrong: a frontier of
one edge, queues of vertices without out-edges (more of them than a tile
stages), one vertex with many edges, ragged ends of tiles and runs, equal
roots; host- and device-driven steps.  The fixpoint does not depend on the
order of the relaxations, so distances equal the single-root ones bit for bit."""
import numpy as np
import pytest

import geminigraph_gb300 as gg

pytestmark = pytest.mark.gpu


def edges(shape, rng):
    if shape == "chain":
        V = 67
        return V, np.arange(V - 1), np.arange(1, V)
    if shape == "star":  # 5000 leaves without out-edges, twice; then a few edges on
        V = 5003
        return V, np.r_[np.zeros(5000), np.zeros(5000), 7, 5001], np.r_[np.arange(1, 5001), np.arange(1, 5001), 5001, 5002]
    if shape == "tiny":
        return 2, np.array([0, 0, 1]), np.array([1, 0, 1])
    V = 3001
    return V, (V * rng.random(40003) ** 2), rng.integers(0, V, 40003)


@pytest.mark.parametrize("device_steps", [False, True])
@pytest.mark.parametrize("shape", ["tiny", "chain", "star", "skewed"])
def test_distances(shape, device_steps):
    rng = np.random.default_rng(5)
    V, s, d = edges(shape, rng)
    s, d = np.asarray(s).astype(np.uint32), np.asarray(d).astype(np.uint32)
    g = gg.Graph.from_edges(V, s, d, rng.random(len(s), dtype=np.float32))
    g.set_batched_graph(device_steps)
    for n, lanes in ((1, 0), (33, 0), (64, 0), (64, 4)):
        g.set_batched_thread_lanes(lanes)
        roots = np.r_[0, 0, rng.integers(0, V, 62)][:n].astype(np.uint32)
        dist, reached, _ = gg.sssp_batched(g, roots)
        for r in sorted(set(roots.tolist())):
            single, _ = g.sssp(r)
            for i in np.flatnonzero(roots == r):
                assert np.array_equal(dist[i].view(np.uint32), single.view(np.uint32)), f"lane {i} root {r}"
                assert int(reached[i]) == int((single < 1e9).sum())
    g.close()
