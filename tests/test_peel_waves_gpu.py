"""Peels in which most of a wave of removals falls to one warp, which keeps at
most 16 vertices while others wait: grids and layered graphs (waves of a few
to thousands of vertices, one to eight entries each); and chains of single
removals, which a warp works off an entry per lane up to 32 entries: lists of
31 to 33, of one side (leaves along the chain) and of both (a chain that falls
out of a row because its end left the core).  Both kinds of instance, against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(n, m):
    i = np.arange(n * m).reshape(n, m)
    return n * m, np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()]), np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])


def layers(width, deg, count):
    rng = np.random.default_rng(width)
    s = np.arange(width * (count - 1)).repeat(deg)
    return width * count, s, (s // width + 1) * width + rng.integers(0, width, len(s))


def leaves(n, deg):
    i = np.arange(n)
    s, d = [i[:-1], i.repeat(deg)], [i[1:], n + np.arange(n * deg)]
    return n * (deg + 1), np.concatenate(s), np.concatenate(d)


def row_chain(n, K):
    """A clique of K + 1, a path into it whose vertices have K in-edges from it,
    the last one two fewer."""
    a, b = np.divmod(np.arange((K + 1) ** 2), K + 1)
    p = np.arange(n) + K + 1
    s, d = [a[a != b], p], [b[a != b], np.append(p[1:], 0)]
    for j in range(K):
        q = p if j < K - 2 else p[:-1]
        s.append(np.full(len(q), j))
        d.append(q)
    return n + K + 1, np.concatenate(s), np.concatenate(d)


CASES = [(grid, (2, 30)), (grid, (15, 40)), (grid, (16, 16)), (grid, (17, 33)), (grid, (300, 300)), (layers, (15, 3, 50)),
         (layers, (17, 1, 200)), (layers, (500, 4, 80)), (layers, (3000, 8, 20)), (grid, (1, 3000)),
         (leaves, (400, 30)), (leaves, (400, 31)), (leaves, (400, 32)), (row_chain, (300, 4)), (row_chain, (300, 29)),
         (row_chain, (300, 30)), (row_chain, (300, 31))]


@pytest.mark.parametrize("make,args", CASES)
def test_peel_waves(dc, orc, gpu, make, args):
    V, s, d = make(*args)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    # a cycle through some vertices: they have core numbers above 0
    ring = np.arange(0, V, max(1, V // 40), dtype=np.uint32)
    s, d = np.concatenate([s, ring]), np.concatenate([d, np.roll(ring, -1)])
    okm, olm, okmaxes, orows = orc.dcore(V, s, d)
    with dc.Graph.from_edges(V, s, d) as g:
        for launch in (1, 4):
            g.set_launch(launch)
            for method in (0, 1):
                assert g.decompose(method) == (okm, olm)
                assert np.array_equal(g.kmaxes(), okmaxes)
                assert np.array_equal(g.rows(), orows)
