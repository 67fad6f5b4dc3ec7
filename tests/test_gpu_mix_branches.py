"""A mixed batch planned with little device memory left (the per-code graph
then has four branches, whose codes share message slabs, instead of sixteen)
gives the results of the plan made with all of it."""
import numpy as np
import pytest

import dvbrx_b200 as D
from test_gpu_mix import CODES, make_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2100])
def test_few_branches(n):
    import torch
    code, llr, handles = make_batch(n, 11)
    for h in handles:
        h.close()
    out = torch.zeros((n, 7290), dtype=torch.uint8, device="cuda")
    it = torch.zeros(n, dtype=torch.int32, device="cuda")
    ok = torch.zeros(n, dtype=torch.uint8, device="cuda")

    def decode():
        mix = D.LdpcMix([(s, r) for s, r, _, _ in CODES])
        mix.plan(code, llr, out, it, ok, 30)
        mix.set_tiling(D.TILING_PER_CODE)
        for t in (out, it, ok):
            t.zero_()
        mix.run()
        torch.cuda.synchronize()
        res = [t.cpu().numpy() for t in (out, it, ok)]
        mix.close()
        return res

    want = decode()
    # 300 frames of each code: about 185 MB of slabs on seven branches, over half of what is left
    torch.cuda.empty_cache()
    fill = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (340 << 20)), dtype=torch.uint8, device="cuda")
    try:
        got = decode()
    finally:
        del fill
        torch.cuda.empty_cache()
    assert want[2].any()
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
