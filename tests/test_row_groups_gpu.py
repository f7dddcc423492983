"""Groups of blocks that run out of rows join others: few rows for many groups,
runs of one row, a core that collapses in its last row, and the same graph
many times over (who joins whom depends on timing); the decomposition equals
the one of a single run and the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def collapse(rng, n, deg, shells):
    """A random directed core of in- and out-degree deg whose members all leave
    at the same row, inside shells of falling degree."""
    e = [np.stack([np.arange(n).repeat(deg), (np.arange(n).repeat(deg) + 1 + np.tile(np.arange(deg), n) * 7) % n], 1)]
    lo = 0
    for k in range(1, shells):
        m = n * 2 * k
        e.append(np.stack([rng.integers(lo, n * (k + 1), m), rng.integers(lo, n * (k + 1), m)], 1))
    return np.concatenate(e)


@pytest.mark.parametrize("cuts", [(10, 20, 30, 40, 50, 60, 70), (500,), (930, 940, 950, 960, 970, 980, 990), (100, 300, 600)])
@pytest.mark.parametrize("kind", ["rmat", "collapse"])
def test_groups_join(dc, orc, gpu, cuts, kind):
    rng = np.random.default_rng(len(cuts))
    if kind == "rmat":
        V, s, d = dc.gen_rmat(13, 32, 51)
    else:
        e = collapse(rng, 1500, 60, 4)
        V, s, d = 6000, e[:, 0].astype(np.uint32), e[:, 1].astype(np.uint32)
    okm, olm, okmaxes, orows = orc.dcore(V, s, d)
    with dc.Graph.from_edges(V, s, d) as one, dc.Graph.from_edges(V, s, d) as g:
        one.set_tuning(2, 2, 64, ())
        assert one.decompose() == (okm, olm)
        want = one.skyline()
        g.set_tuning(2, 2, 64, cuts)
        for turn in range(8):
            assert g.decompose() == (okm, olm)
            assert np.array_equal(g.kmaxes(), okmaxes)
            assert all(np.array_equal(x, y) for x, y in zip(g.skyline(), want))
        assert np.array_equal(g.rows(), orows)
