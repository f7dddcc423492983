"""Text graphs and .decompCPU files around the pieces (1 MiB) they are read and
written in: the device path equals the host parser and writer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PIECE = 1 << 20


@pytest.mark.parametrize("size", [PIECE - 1, PIECE, PIECE + 1, 3 * PIECE + 5])
@pytest.mark.parametrize("newline", [True, False])
def test_file_sizes(dc, gpu, tmp_path, size, newline):
    rng = np.random.default_rng(size)
    V = 3000
    e = rng.integers(0, V, (size // 8, 2))
    text = f"# {V}\n" + "".join(f"{a} {b}\n" for a, b in e.tolist())
    assert len(text) > size
    text = text[:size - 6]
    text = text[:text.rindex("\n") + 1]
    # a last line that ends the file at the wanted size
    last = "1" + " " * (size - len(text) - 2 - newline) + "2" + ("\n" if newline else "")
    p = tmp_path / "g.txt"
    p.write_text(text + last)
    assert p.stat().st_size == size
    n, s, d = dc.read_text_edges(str(p))
    with dc.Graph.load_text_device(str(p)) as g:
        assert g.info() == (n, len(s))
        gs, gd = g.edges()
        x, y = np.lexsort((gd, gs)), np.lexsort((d, s))
        assert np.array_equal(gs[x], s[y]) and np.array_equal(gd[x], d[y])
        g.decompose()
        a, b = tmp_path / "a", tmp_path / "b"
        g.write_decomp_cpu_device(str(a))
        g.write_decomp_cpu(str(b))
        assert a.read_bytes() == b.read_bytes()
