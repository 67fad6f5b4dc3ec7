"""A decode call captured into a CUDA graph allocates nothing when an earlier
call of the handle has already used as much of the device: whichever stopping
rule or entry point that was, its scratch serves the captured call."""
import pytest
import torch

import dvbrx_b200 as D

N = 1000  # more frames than the device holds at once, so both rules fill it


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["group", "host"])
def test_capture_after_another_call(first):
    d = D.Ldpc(D.fec_lookup(0, "3_5"), "3_5")
    llr, _, _ = d.generate(N, 6.5, seed=5, constellation="8PSK")
    if first == "group":
        want = d.decode_device(llr, 30, stop=2)[0]
    else:
        want = torch.from_numpy(d.decode_host(llr.cpu().numpy(), 30)[0]).cuda()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        out, it, ok = d.decode_device(llr, 30, stream=s)
    g.replay()
    torch.cuda.synchronize()
    assert bool((ok == 1).all()) and torch.equal(out, want)
    g.reset()
    d.close()
