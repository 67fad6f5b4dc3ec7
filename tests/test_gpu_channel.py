"""The frame generator: at an Es/N0 without errors its LLR signs are the
codeword of its information bits (the oracle's encoder), for one and several
CTAs per frame, every label width, codes whose parity and information do not
end on words, and an information length short of a byte."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("short,rate,const,const_rate", [
    (0, "1_4", "QPSK", "1_4"), (1, "1_4", "QPSK", "1_4"), (0, "3_5", "8PSK", "3_5"), (1, "2_5", "8PSK", "2_3"),
    (0, "9_10", "16APSK", "9_10"), (1, "8_9", "32APSK", "8_9"), (0, "2_3", "64APSK", "128_180"),
    (0, "5_6", "128APSK", "135_180"), (0, "135_180", "256APSK", "135_180")])
def test_generated_frames_are_codewords(short, rate, const, const_rate):
    code = oracle.OrcCode(short, rate)
    info = D.code_info(short, rate)
    dec = D.Ldpc(D.FecParams(short, info.nldpc, info.K - 3, info.K - 203, 0), rate)  # kldpc not a multiple of 8
    whole = D.Ldpc(D.FecParams(short, info.nldpc, info.K, info.K - 200, 0), rate)
    few = whole.generate(2, 60.0, seed=9, constellation=const, const_rate=const_rate, info=True)
    many = whole.generate(593, 60.0, seed=9, constellation=const, const_rate=const_rate, info=True)
    cut = dec.generate(2, 60.0, seed=9, constellation=const, const_rate=const_rate, info=True)
    assert torch.equal(few[0], many[0][:2]) and torch.equal(few[1], many[1][:2])
    bits = np.unpackbits(few[1].cpu().numpy(), axis=1)[:, : info.K]
    assert np.array_equal((few[0].cpu().numpy() < 0).astype(np.uint8), code.encode(bits))
    assert torch.equal(cut[0], few[0])
    short_bits = np.unpackbits(cut[1].cpu().numpy(), axis=1)
    assert np.array_equal(short_bits[:, : info.K - 3], bits[:, : info.K - 3]) and not short_bits[:, info.K - 3:].any()
    last = whole.generate(593, 5.0, seed=4, constellation=const, const_rate=const_rate, llr_f16=True)
    one = whole.generate(1, 5.0, seed=4, constellation=const, const_rate=const_rate, llr_f16=True)
    assert torch.equal(last[0][0], one[0][0]) and torch.equal(last[2][0], one[2][0])
