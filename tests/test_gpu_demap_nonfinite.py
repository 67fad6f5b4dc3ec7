"""The demapper on symbols that are infinite or not numbers, against the minimum
over the points from infinity on in numpy: a label bit's value whose distances
are all NaN counts as infinitely far, so the other value wins."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
from oracle import datagen

INF, NAN = float("inf"), float("nan")
VALUES = [INF, -INF, NAN, 0.0, 0.7, -1.3]
PAIRS = [(x, y) for x in VALUES for y in VALUES]


def plain_llrs(const, rate, short, sym, n0):
    """Per symbol and label bit: clamp(2/n0 (min_{bit=1} d - min_{bit=0} d)), NaN as -127."""
    bits, order, pts = datagen.constellations()[(const, rate, short)]
    pts = pts / np.sqrt(np.mean(np.abs(pts) ** 2))
    x, y = np.float32([s[0] for s in sym])[:, None], np.float32([s[1] for s in sym])[:, None]
    re, im = np.float32(pts.real), np.float32(pts.imag)
    with np.errstate(all="ignore"):
        d = x * (np.float32(-2.0) * re) + (y * (np.float32(-2.0) * im) + (re * re + im * im))
        out = np.zeros((len(sym), bits), np.float32)
        for b in range(bits):
            one = (np.arange(1 << bits) >> (bits - 1 - b)) & 1 == 1
            m1 = np.fmin.reduce(d[:, one], axis=1, initial=np.float32(np.inf))
            m0 = np.fmin.reduce(d[:, ~one], axis=1, initial=np.float32(np.inf))
            out[:, b] = np.float32(2.0) / np.float32(n0) * (m1 - m0)
    return np.rint(np.clip(np.where(np.isnan(out), -127.0, out), -127.0, 127.0)).astype(int), order


@pytest.mark.gpu
@pytest.mark.parametrize("const,rate,short", [("8PSK", "3_5", 0), ("8PSK", "2_3", 1), ("16APSK", "2_3", 0),
                                              ("32APSK", "3_4", 0), ("64APSK", "128_180", 0)])
@pytest.mark.parametrize("n0", [0.25, -0.25, INF])
@pytest.mark.parametrize("aligned", [True, False])
def test_nonfinite_symbols(const, rate, short, n0, aligned):
    want, order = plain_llrs(const, rate, short, PAIRS, n0)
    dm = D.Demapper(const, rate, short)
    sym = torch.full((dm.nsym, 2), 0.3)
    sym[: len(PAIRS)] = torch.tensor(PAIRS)
    # rows on 16 bytes go to the kernel for whole rows, rows on 8 to the general one
    off = 0 if aligned else 2
    rows = torch.empty(off + 2 * dm.nsym, device="cuda")[off:].view(1, -1)
    rows.copy_(sym.view(1, -1))
    llr = dm.run(rows, torch.tensor([n0], device="cuda"))[0].cpu().numpy().astype(int)
    finite = np.isfinite(np.array(PAIRS)).all(axis=1)
    for b in range(want.shape[1]):
        pos = order[b] * dm.nsym + np.arange(len(PAIRS))
        got = llr[pos]
        assert np.array_equal(got[~finite], want[~finite, b]), b
        # one unit: numpy rounds the products
        assert np.abs(got[finite] - want[finite, b]).max() <= 1
