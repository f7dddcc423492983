"""Lists of the relabeled graph and their support counts at the lengths where
the sort changes (eight lanes with 1, 2 or 4 entries each, a warp, a block, a
counting sort), on either side and at any place of a warp's four lists: all
rows equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 128, 129, 255, 256, 257, 511, 512, 513, 4095, 4096, 4097, 5200]


@pytest.mark.parametrize("pool", [300, 5200])
def test_rows_at_list_lengths(dc, orc, gpu, pool):
    rng = np.random.default_rng(pool)
    hubs = np.arange(len(LENGTHS))
    base = len(LENGTHS)
    # a pool with cores of several depths; hubs over it, out-lists and in-lists of every length
    e = [rng.integers(0, pool // d, (12 * pool // d, 2)) + base for d in (1, 3, 9)]
    for i, n in enumerate(LENGTHS):
        t = np.full(n, i)
        e.append(np.stack([t, base + rng.choice(pool, n, replace=n > pool)], 1))
        m = LENGTHS[-1 - i]
        e.append(np.stack([base + rng.choice(pool, m, replace=m > pool), t[:1].repeat(m)], 1))
    e = np.concatenate(e)
    ids = rng.permutation(base + pool)
    s, d = ids[e[:, 0]].astype(np.uint32), ids[e[:, 1]].astype(np.uint32)
    V = base + pool
    okm, olm, okmaxes, orows = orc.dcore(V, s, d)
    with dc.Graph.from_edges(V, s, d) as g:
        assert g.decompose() == (okm, olm)
        assert np.array_equal(g.kmaxes(), okmaxes)
        assert np.array_equal(g.rows(), orows)
    assert len(hubs) == base and okm > 8
