"""Host-driven deletion batches that take many entries out of single lists:
around a warp's 32, all of a list, its first or last entries only, and
parallel edges of which some stay; the edges left and the decomposition equal
those of the reduced edge list."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def edges_sorted(s, d):
    o = np.lexsort((d, s))
    return np.stack([s[o], d[o]], 1)


@pytest.mark.parametrize("deg,take", [(40, 31), (40, 32), (40, 33), (33, 33), (300, 128), (300, 129), (3000, 2999),
                                      (3000, 3000), (3000, 65)])
@pytest.mark.parametrize("which", ["first", "last", "any"])
def test_many_deletions_of_one_list(dc, orc, gpu, deg, take, which):
    rng = np.random.default_rng(deg + take)
    V = deg + 50
    hub = np.full(deg, V - 1)
    leaf = np.arange(deg)
    rest_s, rest_d = rng.integers(0, V - 1, 600), rng.integers(0, V - 1, 600)
    ok = rest_s != rest_d
    # the hub's out-list, another hub's in-list, every third edge doubled
    s = np.concatenate([hub, hub[::3], leaf, rest_s[ok]]).astype(np.uint32)
    d = np.concatenate([leaf, leaf[::3], np.full(deg, V - 2), rest_d[ok]]).astype(np.uint32)
    keep = s != d
    s, d = s[keep], d[keep]
    pick = {"first": leaf[:take], "last": leaf[deg - take:], "any": rng.permutation(leaf)[:take]}[which]
    ds = np.concatenate([np.full(take, V - 1), pick, rest_s[ok][:40]]).astype(np.uint32)
    dd = np.concatenate([pick, np.full(take, V - 2), rest_d[ok][:40]]).astype(np.uint32)
    k = ds != dd
    ds, dd = ds[k], dd[k]
    left = list(map(tuple, np.stack([s, d], 1).tolist()))
    from collections import Counter
    cnt = Counter(left)
    cnt.subtract(Counter(zip(ds.tolist(), dd.tolist())))
    assert min(cnt.values()) >= 0
    e = np.array(sorted(x for x, m in cnt.items() for _ in range(m)), np.uint32)
    with dc.Graph.from_edges(V, s, d) as g:
        g.decompose()
        st = g.maintain(ds, dd, np.ones(len(ds), np.uint8), 2)
        assert st["deleted"] == len(ds) and st["captured"] == 0
        gs, gd = g.edges()
        assert np.array_equal(edges_sorted(gs, gd), edges_sorted(e[:, 0], e[:, 1]))
        okm, olm, okmaxes, orows = orc.dcore(V, np.ascontiguousarray(e[:, 0]), np.ascontiguousarray(e[:, 1]))
        assert np.array_equal(g.kmaxes(), okmaxes)
        assert np.array_equal(g.rows(), orows)
        # an edge that is not there any more: refused, nothing applied
        with pytest.raises(dc.DCoreError):
            g.maintain(np.r_[e[0, 0], V - 1].astype(np.uint32).repeat(40), np.r_[e[0, 1], V - 1].astype(np.uint32).repeat(40),
                       np.ones(80, np.uint8), 2)
        gs, gd = g.edges()
        assert np.array_equal(edges_sorted(gs, gd), edges_sorted(e[:, 0], e[:, 1]))
