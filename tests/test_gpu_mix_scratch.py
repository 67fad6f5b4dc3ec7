"""A mixed plan whose message memory for sixteen graph branches cannot be had is
made with four branches, with the same results; when that fails too, the plan
fails and a later one works."""
import numpy as np
import pytest

import dvbrx_b200 as D
from test_gpu_mix import CODES, make_batch

ALLOCATIONS_BEFORE = 3  # frame codes, order and counters come before the messages


@pytest.mark.gpu
def test_plan_after_failed_message_allocation():
    import torch
    n = 700
    code, llr, handles = make_batch(n, 12)
    for h in handles:
        h.close()
    out = torch.zeros((n, 7290), dtype=torch.uint8, device="cuda")
    it = torch.zeros(n, dtype=torch.int32, device="cuda")
    ok = torch.zeros(n, dtype=torch.uint8, device="cuda")
    mix = D.LdpcMix([(s, r) for s, r, _, _ in CODES])

    def plan(fail_after=-1):
        D.test_fail_device_alloc(fail_after)
        try:
            mix.plan(code, llr, out, it, ok, 30)
        finally:
            D.test_fail_device_alloc(-1)

    def decode():
        mix.set_tiling(D.TILING_PER_CODE)
        for t in (out, it, ok):
            t.zero_()
        mix.run()
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (out, it, ok)]

    plan()
    assert mix.branches() == 16
    want = decode()
    assert want[2].any()
    plan(ALLOCATIONS_BEFORE)
    assert mix.branches() == 4
    for a, b in zip(want, decode()):
        assert np.array_equal(a, b)
    with pytest.raises(RuntimeError, match="out of memory|memory allocation"):
        plan(0)
    assert mix.branches() == 0
    plan()
    assert mix.branches() == 16
    for a, b in zip(want, decode()):
        assert np.array_equal(a, b)
    mix.close()
