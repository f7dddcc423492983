"""dc_set_launch bounds the row kernel also where the engine cuts the rows: a
launch of one block per SM has no block beyond that.  Shown with the hook that
makes one block of the next launch leave: of 148 blocks the first group holds
two ninths (32), of three blocks per SM 98, so withholding block 40 of the
first group makes the others' waits run out only in a launch that is too wide."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_one_block_per_sm(dc, gpu):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    V, s, d = dc.gen_rmat(16, 40, 7)
    assert len(s) > 1_500_000  # the engine would take all blocks that fit
    with dc.Graph.from_edges(V, s, d) as g:
        K, _ = g.decompose()
        want = g.rows()
        g.set_wait_limit(200_000_000)
        g.set_launch(1)
        g.withhold_barrier(2 * sms // 9 + 8)
        g.decompose_rows(1, K)  # (kmax and row 0 are at hand: the row kernel alone)
        assert np.array_equal(g.rows(1, K), want[1:])
        # two blocks per SM: the same block is one of the first group's
        g.set_launch(2)
        g.withhold_barrier(2 * sms // 9 + 8)
        with pytest.raises(dc.DCoreError) as e:
            g.decompose_rows(1, K)
        assert e.value.code == -6, str(e.value)
        g.decompose_rows(1, K)
        assert np.array_equal(g.rows(1, K), want[1:])
