"""A BCH decode starts from an empty queue whatever an earlier call left behind
in the handle's workspace (a decode that was cut short, calls that overlapped):
all of a batch's words are corrected, and none twice."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
import oracle


@pytest.mark.gpu
@pytest.mark.parametrize("short,rate", [(0, "3_5"), (1, "8_9")])
@pytest.mark.parametrize("left", [1, 37, 1 << 20])
def test_decode_after_left_over_frames(short, rate, left):
    p = D.fec_lookup(short, rate)
    rng = np.random.default_rng(left)
    n = 40
    words = oracle.bch_encode(short, rate, rng.integers(0, 256, (n, p.kbch // 8), dtype=np.uint8))
    sent = words.copy()
    errors = np.arange(n) % (p.t + 1)
    for f in range(n):
        for b in rng.choice(p.kldpc, errors[f], replace=False):
            sent[f, b // 8] ^= 0x80 >> (b % 8)
    bch = D.Bch(p)
    rows = torch.from_numpy(sent).cuda()
    assert np.array_equal(bch.decode_device(rows).cpu().numpy(), errors)  # the workspace exists
    bch.test_left_over(left)
    for k in (n, 7, n):
        rows = torch.from_numpy(sent[:k]).cuda()
        res = bch.decode_device(rows)
        assert np.array_equal(res.cpu().numpy(), errors[:k])
        assert np.array_equal(rows.cpu().numpy(), words[:k])
