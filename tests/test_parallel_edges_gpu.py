"""Multigraphs whose core numbers exceed the number of vertices: per-kmax
arrays are sized by kmax, not by vertices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,m", [(1, 1), (1, 3000), (2, 1), (2, 40), (2, 5000), (3, 700), (40, 90)])
def test_core_numbers_above_vertices(dc, gpu, V, m):
    # every ordered pair (self-loops included) m times: all of C_k, D-core numbers m * V
    u, v = [a.ravel().astype(np.uint32) for a in np.meshgrid(np.arange(V), np.arange(V))]
    with dc.Graph.from_edges(V, np.tile(u, m), np.tile(v, m)) as g:
        km, lm = g.decompose()[:2]
        assert (km, lm) == (m * V, m * V)
        assert (g.kmaxes() == m * V).all()
        rows = g.rows()
        assert rows.shape == (m * V + 1, V) and (rows == m * V).all()
