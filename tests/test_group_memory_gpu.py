"""Cuts that the engine chooses by itself cost memory for the row groups; a
decomposition that has room for one run of rows but not for the groups still
succeeds, with the same result.  The card is filled but for a stretch that is
varied between what one run of this graph wants and what the groups want."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def trim():
    import torch
    from cuda.bindings import runtime as rt
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert err == rt.cudaError_t.cudaSuccess
    assert rt.cudaMemPoolTrimTo(pool, 0)[0] == rt.cudaError_t.cudaSuccess


def attempt(dc, graph, settings, room):
    """A first decomposition of a new handle with `room` bytes left beside the
    graph: its result, or None where memory ran out."""
    import torch
    trim()
    with dc.Graph.from_edges(*graph) as g:
        if settings:
            g.set_tuning(*settings)
        g.synchronize()
        trim()
        ballast = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        try:
            g.decompose()
        except dc.DCoreError as e:
            assert e.code == -3, str(e)
            return None
        finally:
            del ballast
            trim()
        return [g.kmaxes().copy()] + [np.array(x) for x in g.skyline()]


def test_decompose_without_room_for_groups(dc, gpu):
    graph = dc.gen_rmat(20, 8, 2)
    one = (2, 2, 64, ())
    want = attempt(dc, graph, None, 8192 * MIB)
    need = {}
    for name, settings in (("one", one), ("engine", None)):
        with dc.Graph.from_edges(*graph) as g:
            if settings:
                g.set_tuning(*settings)
            before = g.device_bytes()
            g.decompose()
            need[name] = g.device_bytes() - before
    assert need["engine"] > need["one"] + 32 * MIB  # the groups' state
    fits = {}
    for room in range(need["one"] // MIB - 64, need["one"] // MIB + 48, 16):
        for name, settings in (("one", one), ("engine", None)):
            got = attempt(dc, graph, settings, room * MIB)
            fits[name, room] = got is not None
            assert got is None or all(np.array_equal(x, y) for x, y in zip(got, want))
        assert fits["engine", room] or not fits["one", room], fits
    assert not all(fits.values()) and any(fits.values()), fits  # both ends were met
