"""Prefix sums and list starts at the edges of their tiles (1,024 elements) and
of the largest grid: the stored edges, and the skyline built through them,
equal those of the edge list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 1023, 1024, 1025, 2048, 4097, 16 * 148 * 1024 - 1, 16 * 148 * 1024 + 1, 5000003])
def test_list_starts(dc, gpu, V):
    rng = np.random.default_rng(V)
    E = min(6 * V, 200000)
    s, d = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)
    s[-1] = d[-2] = V - 1
    with dc.Graph.from_edges(V, s, d) as g:
        gs, gd = g.edges()
        a, b = np.lexsort((gd, gs)), np.lexsort((d, s))
        assert np.array_equal(gs[a], s[b]) and np.array_equal(gd[a], d[b])
        K, _ = g.decompose()
        off, k, l = g.skyline()[:3]
        km = g.kmaxes()
        assert len(off) == V + 1 and off[0] == 0 and off[-1] == len(k) == len(l) and (np.diff(off.astype(np.int64)) >= 1).all()
        assert (k[off[:-1]] == 0).all()  # each vertex's first corner is row 0
        assert km.max() == K and (km[np.bincount(d, minlength=V) == 0] == 0).all()
