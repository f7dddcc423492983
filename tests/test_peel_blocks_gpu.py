"""The peel's blocks chosen by the number of vertices, on both sides of both
lines: kmax and row 0 as with the blocks set by hand."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [49999, 50000, 50001, 2999999, 3000000])
def test_blocks_by_vertices(dc, gpu, V):
    rng = np.random.default_rng(V)
    E = 4 * V
    # a third of the edges among a hundredth of the vertices
    s, d = rng.integers(0, V, E), rng.integers(0, V, E)
    s[: E // 3], d[: E // 3] = rng.integers(0, V // 100, E // 3), rng.integers(0, V // 100, E // 3)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    with dc.Graph.from_edges(V, s, d) as a, dc.Graph.from_edges(V, s, d) as b:
        assert a.tuning() == b.tuning()
        b.set_tuning(2, 2, 64, ())
        assert a.decompose() == b.decompose()
        assert np.array_equal(a.kmaxes(), b.kmaxes())
        assert all(np.array_equal(x, y) for x, y in zip(a.skyline(), b.skyline()))
