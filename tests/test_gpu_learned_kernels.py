"""The training kernels in every degree class, on layers with few and with
many wavefront levels, against the same decoder in float64 with torch
operations (test_gpu_learned.reference_loss): LLRs from the generator and
LLRs with zeros of both signs, saturated values and ties; one frame and a
batch; posteriors of the forward without training equal the training one's."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
from dvbrx_b200 import learned as L
from test_gpu_learned import reference_loss

pytestmark = pytest.mark.gpu


# degrees 3-4, 4-7, 9-13, 11, 16-19, 27, and normal codes of degree 4 and 22
@pytest.mark.parametrize("short,rate,n", [(1, "1_4", 3), (1, "1_2", 1), (1, "3_4", 2), (1, "3_5", 2), (1, "5_6", 2),
                                          (1, "8_9", 2), (0, "1_4", 1), (0, "5_6", 1)])
@pytest.mark.parametrize("exact_ties", [False, True])
def test_training_kernels_against_float64(short, rate, n, exact_ties):
    iters = 2
    p = D.fec_lookup(short, rate)
    dec = D.Ldpc(p, rate)
    _, info, llr = dec.generate(n, 6.0, seed=3, info=True, llr=False, llr_f16=True)
    g = torch.Generator().manual_seed(1)
    degs, cod = L.degree_classes(short, rate)
    if exact_ties:
        # integers with unit tables: every sum is exact, so ties and clamps fall alike in both
        vals = torch.tensor([-200.0, -128.0, -3.0, -1.0, -0.0, 0.0, 1.0, 3.0, 127.0, 200.0])
        llr = vals[torch.randint(0, 10, (n, dec.N), generator=g)].half().cuda()
        beta0 = alpha0 = torch.ones((iters, len(degs)), device="cuda")
    else:
        beta0 = (0.75 + 0.5 * torch.rand((iters, len(degs)), generator=g)).half().float().cuda()
        alpha0 = (0.25 + torch.rand((iters, len(degs)), generator=g)).half().float().cuda()
    work = L._Work(dec, n, iters, cod)
    b, a = beta0.clone().requires_grad_(True), alpha0.clone().requires_grad_(True)
    loss = L.LearnedMinSum.apply(b, a, dec, llr, info, iters, cod, work)
    loss.backward()
    rb, ra = beta0.double().requires_grad_(True), alpha0.double().requires_grad_(True)
    bits = np.unpackbits(info.cpu().numpy(), axis=1)[:, : p.kldpc]
    want = reference_loss(short, rate, llr.double(), bits, rb, ra, iters, cod)
    want.backward()
    # fp32 sums of a few hundred thousand terms: 1e-4 of the value; gradients 1e-3 of their norm,
    # as the existing comparison
    assert abs(float(loss.detach()) - float(want.detach())) <= 1e-4 * abs(float(want.detach())) + 1e-6
    if not exact_ties:  # topk may route a tie's gradient to another link than the first
        for got, ref in ((b.grad, rb.grad), (a.grad, ra.grad)):
            assert float((got - ref.float()).norm()) <= 1e-3 * float(ref.norm()) + 1e-9
    sums, post = L.learned_posteriors(dec, beta0, alpha0, cod, llr, info, iters)
    assert abs(float(sums.sum()) / (iters * n * p.kldpc) - float(loss.detach())) <= 1e-5 * abs(float(loss.detach()))
    assert post.shape == (n, p.kldpc) and bool(torch.isfinite(post).all())
