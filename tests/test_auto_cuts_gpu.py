"""Cuts chosen by the engine on a handle whose launch shapes were never set:
the same decomposition as one launch for all rows and as the oracle's, where
the cores shrink fast (cut), where they do not (whole), and at the smallest
run of rows that is cut; maintenance that recomputes many rows on such a
handle stays exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graphs(dc):
    yield dc.gen_rmat(13, 32, 21)               # skewed: cut
    yield (2000, *dc.gen_er(2000, 120000, 22))  # every vertex in almost every core: whole
    for extra in (0, 1):                        # complete digraph of 32 / 33: kmax 31 (never cut) and 32
        n = 32 + extra
        u, v = np.meshgrid(np.arange(n), np.arange(n))
        s, d = dc.gen_er(3000, 9000, 23)
        m = (s >= n) | (d >= n)
        yield 3000, np.concatenate([u[u != v], s[m]]).astype(np.uint32), np.concatenate([v[u != v], d[m]]).astype(np.uint32)


def test_fresh_handle_equals_one_launch(dc, orc, gpu):
    for V, s, d in graphs(dc):
        okm, olm, okmaxes, orows = orc.dcore(V, s, d)
        with dc.Graph.from_edges(V, s, d) as a, dc.Graph.from_edges(V, s, d) as b:
            b.set_tuning(2, 2, 64, ())
            assert a.tuning() == b.tuning()
            for g in (a, b):
                assert g.decompose() == (okm, olm)
                assert np.array_equal(g.kmaxes(), okmaxes)
                assert np.array_equal(g.rows(), orows)
            assert all(np.array_equal(x, y) for x, y in zip(a.skyline(), b.skyline()))


def test_maintenance_on_a_fresh_handle(dc, orc, gpu):
    V, s, d = dc.gen_rmat(13, 32, 31)
    u, v, x = dc.gen_updates(V, s, d, 1200, 0.5, 32)
    keys = set(zip(s.tolist(), d.tolist()))
    with dc.Graph.from_edges(V, s, d) as g:
        g.decompose()
        for i in range(0, 1200, 400):
            st = g.maintain(u[i:i + 400], v[i:i + 400], x[i:i + 400])
            for a, b, z in zip(u[i:i + 400].tolist(), v[i:i + 400].tolist(), x[i:i + 400].tolist()):
                keys.discard((a, b)) if z else keys.add((a, b))
            e = np.array(sorted(keys), np.uint32)
            okm, olm, okmaxes, orows = orc.dcore(V, np.ascontiguousarray(e[:, 0]), np.ascontiguousarray(e[:, 1]))
            assert st["rows_recomputed"] > 49
            assert (st["kmax"], st["lmax"]) == (okm, olm)
            assert np.array_equal(g.kmaxes(), okmaxes)
            assert np.array_equal(g.rows(), orows)


@pytest.mark.parametrize("skew", [True, False])
@pytest.mark.parametrize("E", [(8 << 20) - 1, 8 << 20])
def test_cut_rule_by_edges(dc, gpu, skew, E):
    """Both sides of the rule's line at 8 M edges, with every cut allowed
    (skewed degrees) and with the lower ones inside too large a core (a small
    dense part on 12 random edges per vertex)."""
    if skew:
        V, s, d = dc.gen_rmat(19, 18, 41)
    else:
        V, (a, b) = 1 << 19, dc.gen_er(1 << 19, 6 << 20, 42)
        _, u, v = dc.gen_rmat(15, 128, 43)
        s, d = np.concatenate([a, u]), np.concatenate([b, v])
    assert len(s) >= E
    keep = np.random.default_rng(44).permutation(len(s))[:E]
    s, d = np.ascontiguousarray(s[keep]), np.ascontiguousarray(d[keep])
    with dc.Graph.from_edges(V, s, d) as a, dc.Graph.from_edges(V, s, d) as b:
        b.set_tuning(2, 2, 64, ())
        assert a.decompose() == b.decompose()
        assert np.array_equal(a.kmaxes(), b.kmaxes())
        assert all(np.array_equal(x, y) for x, y in zip(a.skyline(), b.skyline()))


@pytest.mark.parametrize("E", [299999, 300000, 1499999, 1500000])
def test_blocks_by_edges(dc, gpu, E):
    """Both sides of the lines between 1, 2 and more blocks per SM for the rows."""
    V, s, d = dc.gen_rmat(16, 32, 45)
    keep = np.random.default_rng(46).permutation(len(s))[:E]
    assert len(keep) == E
    s, d = np.ascontiguousarray(s[keep]), np.ascontiguousarray(d[keep])
    with dc.Graph.from_edges(V, s, d) as a, dc.Graph.from_edges(V, s, d) as b:
        b.set_tuning(2, 2, 64, ())
        assert a.decompose() == b.decompose()
        assert np.array_equal(a.kmaxes(), b.kmaxes())
        assert all(np.array_equal(x, y) for x, y in zip(a.skyline(), b.skyline()))
