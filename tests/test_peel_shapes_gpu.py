"""Fused peel on shapes that reach each of its paths: lists that end just
before, at and after a piece (4 chunks), a hub whose removal removes more
vertices at once than a warp's stack holds, long chains, cascades that widen
and narrow again, and both kinds of instance (kmax and row 0; rows k >= 1 of
the per-row method), against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stars(n):
    """Hub -> n leaves -> one sink, and the reverse of it."""
    h = np.full(n, n)
    s = np.full(n, n + 1)
    leaf = np.arange(n)
    return n + 2, np.concatenate([h, leaf, leaf, s]), np.concatenate([leaf, s, h, leaf])


def hourglass(n):
    """Chains of n vertices that end in hubs, the hubs' leaves in further chains."""
    e, o = [], 0
    for w in (1, 3, 40, 700, 40, 3, 1):
        ids = np.arange(o, o + n * w).reshape(n, w)
        for i in range(n - 1):
            e.append(np.stack([ids[i], ids[i + 1]], 1))
        e.append(np.stack([np.repeat(ids[-1], 20), o + n * w + (np.arange(20 * w) % (n * 3))], 1))
        o += n * w
    e = np.concatenate(e)
    return int(e.max()) + 1, e[:, 0], e[:, 1]


def mixed(n):
    """A core of degree about 30, n vertices hanging off it, and a hub to all."""
    rng = np.random.default_rng(n)
    V = 200 + n + 1
    core = rng.integers(0, 200, (6000, 2))
    hang = np.stack([rng.integers(0, 200, 3 * n), 200 + rng.integers(0, n, 3 * n)], 1)
    back = np.stack([200 + rng.integers(0, n, 2 * n), rng.integers(0, 200, 2 * n)], 1)
    hub = np.stack([np.full(V - 1, V - 1), np.arange(V - 1)], 1)
    e = np.unique(np.concatenate([core, hang, back, hub]), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    return V, e[:, 0], e[:, 1]


CASES = [(stars, n) for n in (1, 63, 64, 65, 255, 256, 257, 1025, 20000)] + \
        [(hourglass, 12), (mixed, 100), (mixed, 1000), (mixed, 30000)]


@pytest.mark.parametrize("chunk", [16, 64])
@pytest.mark.parametrize("make,n", CASES)
def test_peel_shapes(dc, orc, gpu, make, n, chunk):
    V, s, d = make(n)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    okm, olm, okmaxes, orows = orc.dcore(V, s, d)
    with dc.Graph.from_edges(V, s, d) as g:
        g.set_tuning(2, 2, chunk, ())
        for method in (0, 1):
            assert g.decompose(method) == (okm, olm)
            assert np.array_equal(g.kmaxes(), okmaxes)
            assert np.array_equal(g.rows(), orows)
