"""The frame-pair kernel's wavefront level steps (two, three or four, up to
six, and more shared links in a layer) against the one-frame kernel, which
runs every check in full at its own step: inputs that saturate, inputs full of
zeros and equal magnitudes, plain and learned, on codes of every step form."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
from dvbrx_b200 import learned as L

pytestmark = pytest.mark.gpu

# shared links of the codes' layers at most: 2, 2, 4, 4, 5, 6, 6, 7, 8, 9, 12
CODES = [(0, "1_3"), (1, "1_2"), (0, "3_5"), (1, "3_4"), (1, "3_5"), (0, "5_6"), (0, "8_9"), (0, "4_5"), (0, "9_10"),
         (1, "5_6"), (1, "8_9")]


@pytest.mark.parametrize("short,rate", CODES)
def test_level_steps_against_one_frame_kernel(short, rate):
    dec = D.Ldpc(D.fec_lookup(short, rate), rate)
    rng = np.random.default_rng(11)
    n = 7  # an idle lane at the end
    wide = rng.integers(-128, 128, (n, dec.N))
    ties = rng.choice([-3, -1, 0, 0, 1, 3, 127, -128], (n, dec.N))
    llr = torch.from_numpy(np.concatenate([wide, ties]).astype(np.int8)).cuda()
    degs, cod = L.degree_classes(short, rate)
    scale = rng.uniform(0.5, 3.0, (3, len(degs)))
    offset = rng.uniform(-2.0, 3.0, (3, len(degs)))
    dec.set_learned(scale, offset, cod)
    got = {}
    for variant in (D.VARIANT_PAIR, D.VARIANT_FRAME):
        dec.set_variant(variant)
        plain = [t.clone() for it in (1, 2, 5) for t in dec.decode_device(llr, it)]
        learned = [t.clone() for it in (1, 3) for t in dec.decode_learned(llr, it)[:3]]
        got[variant] = plain + learned
    for a, b in zip(got[D.VARIANT_PAIR], got[D.VARIANT_FRAME]):
        assert torch.equal(a, b)
