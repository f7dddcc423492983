"""The peel of small graphs, one block per peel: kmax and row 0 equal those of
the grid's peel (shapes set by hand) and of the oracle, at its largest V and E,
with one vertex, lists around 32 and 256 entries, more long lists than one
round holds, parallel edges and self-loops, and a chain as long as the graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(kind):
    rng = np.random.default_rng(7)
    if kind == "one":
        return 1, np.zeros(3, int), np.zeros(3, int)
    if kind == "empty":
        return 700, np.zeros(0, int), np.zeros(0, int)
    if kind == "chain":  # removed one by one
        return 3000, np.arange(2999), np.arange(1, 3000)
    if kind == "lists":  # lists of 0..300 entries, out of a ring that holds them up
        n = np.arange(301)
        s = np.concatenate([n.repeat(n), np.arange(301)])
        d = np.concatenate([rng.integers(0, 301, n.sum()), (np.arange(301) + 1) % 301])
        return 301, s, d
    if kind == "hubs":  # 200 lists of 257..1,500 entries removed in the same round
        s = np.arange(200).repeat(rng.integers(257, 1500, 200))
        return 4000, s, 200 + rng.integers(0, 3800, len(s))
    if kind.startswith("even"):  # degrees alike: the line lies lower
        V, E = {"even V": (16384, 200000), "even V+1": (16385, 200000), "even E": (9000, 500000),
                "even E+1": (9000, 500001)}[kind]
        return V, rng.integers(0, V, E), rng.integers(0, V, E)
    V, E = {"V-1": (35999, 300000), "V": (36000, 300000), "V+1": (36001, 300000), "E": (9000, 2000000),
            "E+1": (9000, 2000001)}[kind]
    s, d = rng.integers(0, V, E), rng.integers(0, V, E)
    s[: E // 3], d[: E // 3] = rng.integers(0, V // 50, E // 3), rng.integers(0, V // 50, E // 3)
    return V, s, d


@pytest.mark.parametrize("kind", ["one", "empty", "chain", "lists", "hubs", "V-1", "V", "V+1", "E", "E+1", "even V",
                                  "even V+1", "even E", "even E+1"])
def test_small_peel(dc, orc, gpu, kind):
    V, s, d = graph(kind)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    with dc.Graph.from_edges(V, s, d) as a, dc.Graph.from_edges(V, s, d) as b:
        b.set_tuning(2, 2, 64, ())
        assert a.decompose_rows(0, 0) == b.decompose_rows(0, 0)
        assert a.decompose() == b.decompose()
        assert np.array_equal(a.kmaxes(), b.kmaxes())
        assert np.array_equal(a.rows(0, 1), b.rows(0, 1))
        assert all(np.array_equal(x, y) for x, y in zip(a.skyline(), b.skyline()))
        if len(s) and len(s) < 400000 and V > 1:
            okm, olm, okmaxes, orows = orc.dcore(V, s, d)
            assert (okm, olm) == a.decompose()
            assert np.array_equal(a.kmaxes(), okmaxes) and np.array_equal(a.rows(), orows)
