"""Row kernel at the sizes where its reads change shape: lists that end just
before, at and after a window of 128 entries (and at any 16-byte alignment),
values that fall by less and by more than the register counters cover, and
many vertices leaving at once, against the oracle, whole and cut."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cliques(sizes, extra, seed):
    """Disjoint complete digraphs, every vertex of one with edges into the next
    (so that a clique's collapse takes many out-neighbours away at once), and
    `extra` random edges."""
    rng = np.random.default_rng(seed)
    V = int(sum(sizes)) + 7
    e, o, prev = [], 0, None
    for n in sizes:
        ids = np.arange(o, o + n)
        u, v = np.meshgrid(ids, ids)
        e.append(np.stack([u[u != v], v[u != v]], 1))
        if prev is not None:
            k = min(len(prev), len(ids), 40)
            u, v = np.meshgrid(prev, ids[:k])
            e.append(np.stack([u.ravel(), v.ravel()], 1))
        prev, o = ids, o + n
    r = rng.integers(0, V, (extra, 2))
    e.append(r[r[:, 0] != r[:, 1]])
    e = np.unique(np.concatenate(e), axis=0)
    perm = rng.permutation(V)
    return V, perm[e[:, 0]].astype(np.uint32), perm[e[:, 1]].astype(np.uint32)


@pytest.mark.parametrize("cuts", [(), (100, 300, 500, 700, 900)])
@pytest.mark.parametrize("sizes", [(2, 3, 5), (31, 32, 33), (127, 128, 129, 130), (255, 257, 40), (300, 8, 120, 4)])
def test_list_windows(dc, orc, gpu, sizes, cuts):
    V, s, d = cliques(sizes, 3 * sum(sizes), sum(sizes))
    _, _, okmaxes, orows = orc.dcore(V, s, d)
    with dc.Graph.from_edges(V, s, d) as g:
        g.set_tuning(2, 2, 64, cuts)
        g.decompose()
        assert np.array_equal(g.kmaxes(), okmaxes)
        assert np.array_equal(g.rows(), orows)


def test_many_leavers(dc, orc, gpu):
    """Ten thousand vertices of kmax 1 and 2 around a core leave in two rows."""
    rng = np.random.default_rng(3)
    V0, s, d = cliques((60, 30), 200, 9)
    n = 20000
    new = np.arange(V0, V0 + n)
    core = rng.integers(0, V0, (n, 6))
    s = np.concatenate([s, np.repeat(new, 4), core[:, 4], core[:, 5][: n // 2]]).astype(np.uint32)
    d = np.concatenate([d, core[:, :4].ravel(), new, new[: n // 2]]).astype(np.uint32)
    e = np.unique(np.stack([s, d], 1), axis=0)
    s, d = np.ascontiguousarray(e[:, 0]), np.ascontiguousarray(e[:, 1])
    _, _, okmaxes, orows = orc.dcore(V0 + n, s, d)
    with dc.Graph.from_edges(V0 + n, s, d) as g:
        g.decompose()
        assert np.array_equal(g.kmaxes(), okmaxes)
        assert np.array_equal(g.rows(), orows)


def test_list_sizes(dc, orc, gpu):
    """Out-lists and in-lists of every size where the list sorts change method
    or padding, over neighbours of many different kmax; the edges given grouped
    by source, shuffled, and with parallel edges."""
    rng = np.random.default_rng(11)
    sizes = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1025, 2047, 2049, 4095, 4096,
             4097, 9000]
    V0 = 9500
    V = V0 + 2 * len(sizes)
    e = [rng.integers(0, 60, (2500, 2)), rng.integers(0, 700, (14000, 2)), rng.integers(0, V0, (30000, 2))]
    for i, n in enumerate(sizes):
        pick = rng.permutation(V0)[:n]
        e.append(np.stack([np.full(n, V0 + 2 * i), pick], 1))
        e.append(np.stack([pick[::-1], np.full(n, V0 + 2 * i + 1)], 1))
        e.append(np.array([[V0 + 2 * i + 1, V0 + 2 * i], [pick[0], V0 + 2 * i]]))
    e = np.unique(np.concatenate(e), axis=0)
    e = e[e[:, 0] != e[:, 1]].astype(np.uint32)
    doubled = np.concatenate([e, e[::50], e[::50]])
    for edges in (e, e[rng.permutation(len(e))], doubled[rng.permutation(len(doubled))]):
        s, d = np.ascontiguousarray(edges[:, 0]), np.ascontiguousarray(edges[:, 1])
        _, _, okmaxes, orows = orc.dcore(V, s, d)
        with dc.Graph.from_edges(V, s, d) as g:
            g.decompose()
            assert np.array_equal(g.kmaxes(), okmaxes)
            assert np.array_equal(g.rows(), orows)
            gs, gd = g.edges()
            o, q = np.lexsort((d, s)), np.lexsort((gd, gs))
            assert np.array_equal(gs[q], s[o]) and np.array_equal(gd[q], d[o])
