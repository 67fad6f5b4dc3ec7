"""The demapper's two kernels (rows that are all aligned and whole, and any
rows) against the numpy demapper of oracle.datagen and against each other,
bit for bit between the kernels: every label width, with values that are not
numbers and a noise power near zero."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
from oracle import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("const,rate,short", [
    ("QPSK", "1_2", 0), ("QPSK", "1_2", 1), ("8PSK", "3_5", 0), ("8PSK", "2_3", 1), ("16APSK", "2_3", 0),
    ("16APSK", "8_9", 1), ("32APSK", "3_4", 0), ("32APSK", "5_6", 1), ("64APSK", "128_180", 0),
    ("128APSK", "135_180", 0), ("256APSK", "20_30", 0), ("256APSK", "135_180", 0)])
@pytest.mark.parametrize("n", [1, 3, 70])
def test_demapper_rows(const, rate, short, n):
    dm = D.Demapper(const, rate, short)
    g = torch.Generator(device="cuda").manual_seed(n)
    sym = torch.randn((n, 2 * dm.nsym), generator=g, device="cuda") * 0.8
    n0 = 10.0 ** (-torch.rand(n, generator=g, device="cuda") * 1.5)
    whole = dm.run(sym, n0)
    want = datagen.demap(sym.cpu().numpy().view(np.complex64), n0.cpu().numpy()[:, None], const, rate, short, dm.nldpc)
    diff = np.abs(whole.cpu().numpy().astype(int) - want)
    # the numpy distances round each product: one unit on rare ties
    assert diff.max() <= 1 and (diff != 0).mean() < 2e-3
    sym[0, 5], sym[0, 8], sym[0, 10:12] = float("nan"), float("inf"), 0.0
    n0[-1] = 1e-30
    ref = dm.run(sym, n0)
    for off, stride, out_off, out_stride in ((2, 2 * dm.nsym + 2, 0, dm.nldpc), (0, 2 * dm.nsym, 3, dm.nldpc + 5),
                                             (4, 2 * dm.nsym + 8, 8, dm.nldpc + 16)):
        rows = torch.empty(off + n * stride, device="cuda")[off:].view(n, stride)
        rows[:, : 2 * dm.nsym] = sym
        out = torch.full((out_off + n * out_stride,), 99, dtype=torch.int8, device="cuda")
        llr = out[out_off:].view(n, out_stride)
        dm.run(rows, n0, llr=llr)
        assert torch.equal(llr[:, : dm.nldpc], ref)
        assert bool((llr[:, dm.nldpc:] == 99).all()) and bool((out[:out_off] == 99).all())
