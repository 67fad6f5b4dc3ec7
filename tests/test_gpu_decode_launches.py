"""The kernel count that a device batch is reported to have: two where the frames
are put in order first (per-frame stopping, normal frames, more of them than the
device holds at once, up to 16384, enough iterations for frames to differ)."""
import pytest
import torch

import dvbrx_b200 as D


@pytest.mark.gpu
def test_decode_launches():
    d = D.Ldpc(D.fec_lookup(0, "3_5"), "3_5")
    lanes = 4 * torch.cuda.get_device_properties(0).multi_processor_count  # two CTAs of two frames
    assert [d.decode_launches(n, 30) for n in (0, 1, lanes, lanes + 1, 16384, 16385)] == [0, 1, 1, 2, 2, 1]
    assert d.decode_launches(4096, 7) == 1 and d.decode_launches(4096, 8) == 2
    assert d.decode_launches(4096, 30, stop=64) == 1 and d.decode_launches(4096, 30, stop=-1) == -1
    assert d.set_variant(D.VARIANT_FRAME) == D.VARIANT_FRAME and d.decode_launches(4096, 30) == 1
    d.close()
    s = D.Ldpc(D.fec_lookup(1, "1_2"), "1_2")
    assert s.decode_launches(4096, 30) == 1
    s.close()
