"""The pages of result arrays that a call makes ready before it copies: what
lies in the caller's memory outside the result stays as it was, for results at
any offset in a page, on fresh and on used memory, small and large."""
import ctypes
import mmap

import numpy as np
import pytest

import geminigraph_gb300 as gg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [3, 20011, 300007, 4000003])
def test_only_the_result_is_written(V):
    rng = np.random.default_rng(V)
    s, d = rng.integers(0, V, 2 * V, dtype=np.uint32), rng.integers(0, V, 2 * V, dtype=np.uint32)
    g = gg.Graph.from_edges(V, s, d)
    want, _ = g.cc()
    for offset, fill in ((0, 0), (4, 0), (65536 - 4, 0x5a), (100, 0x5a)):
        m = mmap.mmap(-1, 4 * V + 3 * 65536)
        whole = np.frombuffer(m, np.uint8)
        if fill:
            whole[:] = fill
        out = whole[offset:offset + 4 * V].view(np.uint32)
        rc = gg.library().gg_cc(g.h, ctypes.c_void_p(out.ctypes.data), None)
        assert rc == 0
        assert np.array_equal(out, want)
        assert (whole[:offset] == fill).all() and (whole[offset + 4 * V:] == fill).all()
        del out, whole
        m.close()
    g.close()
