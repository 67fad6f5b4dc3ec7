"""The training kernels of the remaining compiled degrees (the normal codes') and
degree classes (codes with two check degrees) against the same decoder in
float64, loss and gradients; small and large scales, so that magnitudes, clamps
and messages beyond the stored range occur."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
from dvbrx_b200 import learned as L
from test_gpu_learned import reference_loss


# degrees 5, 6, 7, 10, 14, 18, 30 compiled apart; classes by two degrees: 5, 11, 12, 17, 20, 30; 9 in a class
@pytest.mark.gpu
@pytest.mark.parametrize("rate", ["1_3", "2_5", "1_2", "2_3", "3_4", "4_5", "9_10", "13_45", "18_30", "116_180",
                                  "135_180", "140_180", "154_180", "26_45"])
def test_training_degrees_against_float64(rate):
    iters, n = 2, 1
    p = D.fec_lookup(0, rate)
    dec = D.Ldpc(p, rate)
    _, info, llr = dec.generate(n, 6.0, seed=9, const_rate="1_2", info=True, llr=False, llr_f16=True)
    g = torch.Generator().manual_seed(len(rate))
    degs, cod = L.degree_classes(0, rate)
    beta0 = (0.6 + 0.8 * torch.rand((iters, len(degs)), generator=g)).half().float().cuda()
    alpha0 = (2.0 * torch.rand((iters, len(degs)), generator=g) - 0.5).half().float().cuda()
    work = L._Work(dec, n, iters, cod)
    b, a = beta0.clone().requires_grad_(True), alpha0.clone().requires_grad_(True)
    loss = L.LearnedMinSum.apply(b, a, dec, llr, info, iters, cod, work)
    loss.backward()
    rb, ra = beta0.double().requires_grad_(True), alpha0.double().requires_grad_(True)
    bits = np.unpackbits(info.cpu().numpy(), axis=1)[:, : p.kldpc]
    want = reference_loss(0, rate, llr.double(), bits, rb, ra, iters, cod)
    want.backward()
    # as the other comparisons with float64: 1e-4 of the loss, 1e-3 of the gradients' norm
    assert abs(float(loss.detach()) - float(want.detach())) <= 1e-4 * abs(float(want.detach())) + 1e-6
    for got, ref in ((b.grad, rb.grad), (a.grad, ra.grad)):
        assert float(ref.norm()) > 0
        assert float((got - ref.float()).norm()) <= 1e-3 * float(ref.norm()) + 1e-9
    dec.close()
