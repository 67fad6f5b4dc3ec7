"""Batches of more normal frames than the device's lanes are decoded weakest
LLRs first: every frame's results equal those of the same frame in a batch of
few frames (decoded in row order), for row strides of every alignment, frames
of very different and of equal LLR magnitudes, and the largest ordered batch."""
import pytest

import dvbrx_b200 as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,const,es,n,pad,kind", [
    ("3_5", "8PSK", 6.2, 593, 0, "mixed"),
    ("2_3", "8PSK", 7.0, 1025, 1, "mixed"),
    ("9_10", "QPSK", 6.8, 700, 7, "mixed"),
    ("1_4", "QPSK", -1.5, 777, 16, "equal"),
    ("9_10", "QPSK", 7.5, 16384, 0, "extreme"),
])
def test_order_changes_no_result(rate, const, es, n, pad, kind):
    import torch
    dec = D.Ldpc(D.fec_lookup(0, rate), rate)
    m = min(n, 300)
    base, _, _ = dec.generate(m, es, seed=5, constellation=const)
    llr = torch.zeros((n, dec.N + pad), dtype=torch.int8, device="cuda")
    for i in range(0, n, m):
        k = min(m, n - i)
        llr[i:i + k, :dec.N] = base[:k]
    if kind == "mixed":  # the frames' magnitudes differ, some are zero
        llr[1::3, :dec.N] = (llr[1::3, :dec.N].float() * 0.5).to(torch.int8)
        llr[5::50, :dec.N] = 0
    if kind == "extreme":
        llr[3::7] = -128
        llr[4::7] = 127
    got = dec.decode_device(llr, 12)
    torch.cuda.synchronize()
    step = 256
    for i in range(0, n, step):
        want = dec.decode_device(llr[i:i + step], 12)
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a[i:i + step], b), i
    dec.close()
