"""Net effect of batches around the size from which it is taken on the device
(4,096 updates), tiles of its sorts and scans included: repeated, cancelling
and parallel updates in any order; the edges left and the decomposition equal
those of the edge list with the same updates applied."""
from collections import Counter

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def updates(rng, V, present, b):
    """b updates whose net effect deletes only what is there."""
    n_toggle, n_del = b // 4, b // 4
    t = np.stack([rng.integers(0, V, n_toggle), rng.integers(0, V, n_toggle)], 1)
    dele = present[rng.permutation(len(present))[:n_del]]
    n_ins = b - 2 * n_toggle - n_del
    ins = np.stack([rng.integers(0, V, n_ins), rng.integers(0, V, n_ins)], 1)
    ins[: n_ins // 3] = ins[rng.integers(0, max(n_ins // 8, 1), n_ins // 3)]  # parallel edges
    pairs = np.concatenate([t, t, dele, ins])
    flag = np.concatenate([np.zeros(n_toggle), np.ones(n_toggle), np.ones(n_del), np.zeros(n_ins)]).astype(np.uint8)
    o = rng.permutation(b)
    return pairs[o].astype(np.uint32), flag[o]


@pytest.mark.parametrize("V", [1, 2, 60, 1025, 70000])
@pytest.mark.parametrize("b", [4095, 4096, 4097, 6144, 20481])
def test_net_batch(dc, orc, gpu, V, b):
    rng = np.random.default_rng(V + b)
    E = 12000
    s, d = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)
    cnt = Counter(zip(s.tolist(), d.tolist()))
    with dc.Graph.from_edges(V, s, d) as g:
        g.decompose()
        for _ in range(2):
            present = np.array([x for x, m in cnt.items() for _ in range(m)], np.int64)
            pairs, flag = updates(rng, V, present, b)
            for (u, v), f in zip(pairs.tolist(), flag.tolist()):
                cnt[(u, v)] += -1 if f else 1
            assert min(cnt.values()) >= 0
            g.maintain(np.ascontiguousarray(pairs[:, 0]), np.ascontiguousarray(pairs[:, 1]), flag, 2)
        e = np.array(sorted(x for x, m in cnt.items() for _ in range(m)), np.uint32)
        es, ed = np.ascontiguousarray(e[:, 0]), np.ascontiguousarray(e[:, 1])
        gs, gd = g.edges()
        o = np.lexsort((gd, gs))
        assert np.array_equal(gs[o], es) and np.array_equal(gd[o], ed)
        if V > 1 and len(es) <= 60000:
            _, _, okmaxes, orows = orc.dcore(V, es, ed)
            assert np.array_equal(g.kmaxes(), okmaxes)
            assert np.array_equal(g.rows(), orows)


@pytest.mark.parametrize("b", [4095, 4096, 9000])
def test_refused_batches(dc, gpu, b):
    """An id out of range or a missing edge anywhere: refused, nothing applied."""
    rng = np.random.default_rng(b)
    V = 500
    s, d = rng.integers(0, V, 9000).astype(np.uint32), rng.integers(0, V, 9000).astype(np.uint32)
    with dc.Graph.from_edges(V, s, d) as g:
        g.decompose()
        km, before = g.kmaxes().copy(), np.stack(g.edges())
        u, v = rng.integers(0, V, b).astype(np.uint32), rng.integers(0, V, b).astype(np.uint32)
        w = u.copy()
        w[b - 7] = V
        with pytest.raises(dc.DCoreError, match=f"edge {b - 7} .*vertex id >= V={V}"):
            g.maintain(w, v, np.zeros(b, np.uint8), 2)
        f = np.zeros(b, np.uint8)
        present = set(zip(s.tolist(), d.tolist())) | set(zip(u.tolist(), v.tolist()))
        miss = next((x, y) for x in range(V) for y in range(V) if (x, y) not in present)
        u[b // 2], v[b // 2], f[b // 2] = miss[0], miss[1], 1
        with pytest.raises(dc.DCoreError, match="not in the graph"):
            g.maintain(u, v, f, 2)
        assert np.array_equal(np.stack(g.edges()), before) and np.array_equal(g.kmaxes(), km)
        # updates that cancel: nothing changes
        half = b // 2
        g.maintain(np.r_[u[:half], u[:half]], np.r_[v[:half], v[:half]],
                   np.r_[np.zeros(half, np.uint8), np.ones(half, np.uint8)], 2)
        assert np.array_equal(np.stack(g.edges()), before) and np.array_equal(g.kmaxes(), km)


@pytest.mark.parametrize("b", [1 << 20, (1 << 20) + 1, (1 << 20) + 4097])
def test_large_batches(dc, gpu, b):
    """Around a million updates, where the sort's tiles change; few of them
    are left after the others cancel."""
    rng = np.random.default_rng(b)
    V, E = 5000, 30000
    s, d = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)
    gone = rng.permutation(E)[:300]
    n_ins = 200 + (b - 500) % 2
    n = (b - 300 - n_ins) // 2
    t, ins = rng.integers(0, V, (n, 2)), rng.integers(0, V, (n_ins, 2))
    pairs = np.concatenate([t, np.stack([s[gone], d[gone]], 1), ins, t]).astype(np.uint32)
    flag = np.concatenate([np.zeros(n), np.ones(300), np.zeros(n_ins), np.ones(n)]).astype(np.uint8)
    o = rng.permutation(len(pairs))
    assert len(pairs) == b
    with dc.Graph.from_edges(V, s, d) as g:
        g.decompose()
        st = g.maintain(pairs[o, 0], pairs[o, 1], flag[o], 2)
        both = Counter(map(tuple, pairs[n:n + 300].tolist())) & Counter(map(tuple, ins.tolist()))
        assert st["deleted"] == 300 - sum(both.values()) and st["inserted"] == n_ins - sum(both.values())
        keep = np.ones(E, bool)
        keep[gone] = False
        es = np.concatenate([s[keep], ins[:, 0].astype(np.uint32)])
        ed = np.concatenate([d[keep], ins[:, 1].astype(np.uint32)])
        gs, gd = g.edges()
        x, y = np.lexsort((gd, gs)), np.lexsort((ed, es))
        assert np.array_equal(gs[x], es[y]) and np.array_equal(gd[x], ed[y])
