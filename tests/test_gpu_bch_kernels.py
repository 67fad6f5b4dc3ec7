"""The BCH kernels (half-warp and warp remainders, the correction kernel's
locator and root search) against a plain decoder in Python on the code's own
definition: every parity length (t = 8, 10, 12 over GF(2^16), 12 over
GF(2^14)), rows at every byte alignment, batches on both sides of the
remainder kernel's switch, words with 0 .. t + 3 errors and random words."""
import numpy as np
import pytest
import torch

import dvbrx_b200 as D
import oracle

pytestmark = pytest.mark.gpu

SWITCH = 16 * 148  # frames up to which a warp takes one frame (on 148 SMs)


class Field:
    def __init__(self, m):
        self.q = (1 << m) - 1
        prim = 0x1002D if m == 16 else 0x402B
        self.exp, self.log = np.zeros(2 * self.q, np.int64), np.zeros(self.q + 1, np.int64)
        x = 1
        for i in range(self.q):
            self.exp[i] = self.exp[i + self.q] = x
            self.log[x] = i
            x = x << 1
            if x >> m:
                x ^= prim

    def mul(self, a, b):
        return int(self.exp[self.log[a] + self.log[b]]) if a and b else 0


def plain_decode(F, p, word):
    """Corrected bit count or -1, and the word: syndromes, Berlekamp-Massey,
    every position tried."""
    n, t = p.kldpc, p.t
    deg = n - 1 - np.nonzero(np.unpackbits(word)[:n])[0]
    S = [0] + [int(np.bitwise_xor.reduce(F.exp[deg * j % F.q])) if deg.size else 0 for j in range(1, 2 * t + 1)]
    if not any(S):
        return 0, word
    L, B, length, shift, b = [1], [1], 0, 1, 1
    for k in range(2 * t):
        d = S[k + 1]
        for i in range(1, min(length, len(L) - 1) + 1):
            d ^= F.mul(L[i], S[k + 1 - i])
        if not d:
            shift += 1
            continue
        c = F.mul(d, int(F.exp[F.q - F.log[b]]))
        new = L + [0] * (len(B) + shift - len(L))
        for i, v in enumerate(B):
            new[i + shift] ^= F.mul(c, v)
        if 2 * length <= k:
            L, B, length, shift, b = new, L, k + 1 - length, 1, d
        else:
            L, shift = new, shift + 1
    if length > t:
        return -1, word
    pos = np.arange(n)
    v = np.zeros(n, np.int64)
    for i, c in enumerate(L):
        if c:
            v ^= F.exp[(F.log[c] + (F.q - i) * pos) % F.q]
    roots = np.nonzero(v == 0)[0]
    if roots.size != length:
        return -1, word
    out = np.unpackbits(word)
    out[n - 1 - roots] ^= 1
    return length, np.packbits(out)


@pytest.mark.parametrize("short,rate,n", [(0, "3_5", 40), (0, "2_3", 40), (0, "9_10", 40), (0, "1_4", 40),
                                          (1, "1_4", 40), (1, "8_9", 40), (0, "8_9", SWITCH), (0, "1_4", SWITCH + 1),
                                          (1, "2_3", SWITCH + 1), (0, "5_6", 1)])
def test_bch_kernels_against_plain_decoder(short, rate, n):
    p = D.fec_lookup(short, rate)
    F = Field(14 if short else 16)
    rng = np.random.default_rng(n + len(rate))
    few = min(n, 32)  # frames the plain decoder repeats; the others repeat them in turn
    words = oracle.bch_encode(short, rate, rng.integers(0, 256, (few, p.kbch // 8), dtype=np.uint8))
    clean = words.copy()
    for f in range(few):
        for b in rng.choice(p.kldpc, f % (p.t + 4), replace=False):
            words[f, b // 8] ^= 0x80 >> (b % 8)
    if few > 2:
        words[-2:] = rng.integers(0, 256, (2, p.kldpc // 8), dtype=np.uint8)
    want = [plain_decode(F, p, w) for w in words]
    nb = p.kldpc // 8
    bch = D.Bch(p)
    idx = np.arange(n) % few
    for off in (0, 1, 6, 13):
        stride = nb + 3 + off
        buf = torch.full((off + n * stride + 16,), 0xA5, dtype=torch.uint8, device="cuda")
        rows = buf[off:off + n * stride].view(n, stride)
        # encoding: the parity of the clean words, every other byte untouched
        rows[:, : p.kbch // 8] = torch.from_numpy(clean[idx, : p.kbch // 8]).cuda()
        bch.encode_device(rows)
        assert np.array_equal(rows[:, :nb].cpu().numpy(), clean[idx])
        assert bool((rows[:, nb:] == 0xA5).all()) and bool((buf[:off] == 0xA5).all())
        # decoding, twice on one handle (the queue is left empty)
        for _ in range(2):
            rows[:, :nb] = torch.from_numpy(words[idx]).cuda()
            res = bch.decode_device(rows)
            assert np.array_equal(res.cpu().numpy(), np.array([want[k][0] for k in idx], np.int32))
            assert np.array_equal(rows[:, :nb].cpu().numpy(), np.stack([want[k][1] for k in idx]))
            assert bool((rows[:, nb:] == 0xA5).all()) and bool((buf[:off] == 0xA5).all())


@pytest.mark.parametrize("kbytes,stride", [(7274, 7300), (2025, 2025), (17, 64), (5, 33), (0, 8)])
def test_descrambler_at_every_alignment(kbytes, stride):
    from dvbrx_b200.tables.gen_bb import prbs_bytes

    prbs = np.array(prbs_bytes(7274), np.uint8)
    n = 5
    for off in range(17):
        buf = torch.randint(0, 256, (off + n * stride + 16,), dtype=torch.uint8, device="cuda")
        want = buf.cpu().numpy()
        D.bb_descramble(buf[off:off + n * stride].view(n, stride), kbytes)
        want[off:off + n * stride].reshape(n, stride)[:, :kbytes] ^= prbs[:kbytes]
        assert np.array_equal(buf.cpu().numpy(), want), off
