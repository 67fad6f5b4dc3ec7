"""Performance cases: the work a user of this library has it do, through its
public entry points, over the sizes it meets.

Every case is a dict of plain values with a ``kind``:

dropin    ``Ldpc.decode``, the reference receiver's call: up to 64 frames on
          host memory, one call, all frames iterate until all pass.
decode    ``Ldpc.decode_device``: a device batch, per-frame stopping (stop 0)
          or groups of ``stop`` frames.
host      ``Ldpc.decode_host`` on page-locked host rows, in and out.
mixed     ``LdpcMix``: a planned and tuned batch over many codes, replayed.
learned   ``Ldpc.decode_learned``: the committed learned tables with the plain
          decoder for the frames that fail.
train     one training step of ``learned.LearnedDecoder``: the loss (forward)
          and the gradients of the tables (backward).
outer     the stages after LDPC: BCH decoding in place, BBFRAME descrambling
          and the BBHEADER check.
encode    ``Bch.encode_device``: BCH parity of message rows, in place.
demap     ``Demapper.run``: received symbols to int8 LLRs.
generate  ``Ldpc.generate``: seeded frames (encoder, mapper, noise, demapper).

Es/N0 is the MODCOD's quasi-error-free value plus a margin in dB (``margin``
is the highest; frames spread down to ``margin_lo``), where a receiver works.
"""
import functools
import os
import re

import numpy as np
import torch

import dvbrx_b200 as D
from dvbrx_b200 import learned as L
from dvbrx_b200 import modcods as MC
from dvbrx_b200 import train as T

HERE = os.path.dirname(os.path.abspath(__file__))
SPREAD = 7  # Es/N0 points a batch is spread over, as in the benchmark's sweep


def listed():
    return [
        # a receiver that waits for each frame: one short frame per call, latency alone
        {"name": "dropin_short_1", "kind": "dropin", "short": 1, "rate": "1_2", "const": "QPSK", "margin": 1.0,
         "margin_lo": 1.0, "frames": 1, "max_iter": 50},
        # the reference receiver's own call: 64 normal frames per call on host memory
        {"name": "dropin_normal_64", "kind": "dropin", "short": 0, "rate": "3_5", "const": "8PSK", "margin": 0.5,
         "margin_lo": 0.5, "frames": 64, "max_iter": 30},
        # a device batch of short frames (the 1024-frame QPSK 1/2 configuration), one frame short of even
        {"name": "short_1_2_1023", "kind": "decode", "short": 1, "rate": "1_2", "const": "QPSK", "margin": 0.8,
         "margin_lo": 0.2, "frames": 1023, "max_iter": 50, "stop": 0},
        # the benchmark's workload: normal 3/5 8PSK through its waterfall, 4096 frames
        {"name": "normal_3_5_4096", "kind": "decode", "short": 0, "rate": "3_5", "const": "8PSK", "margin": 1.0,
         "margin_lo": -0.5, "frames": 4096, "max_iter": 30, "stop": 0},
        # the same from host memory, end to end, a batch that fills no wave evenly
        {"name": "host_3_5_1777", "kind": "host", "short": 0, "rate": "3_5", "const": "8PSK", "margin": 1.0,
         "margin_lo": -0.5, "frames": 1777, "max_iter": 30},
        # an adaptive-coding carrier: 21 codes in one planned batch
        {"name": "mixed_2048", "kind": "mixed", "frames": 2048, "max_iter": 30},
        # the learned decoder with its fallback, normal 2/3 8PSK at 20 iterations
        {"name": "learned_2_3_1024", "kind": "learned", "short": 0, "rate": "2_3", "const": "8PSK", "margin": 0.5,
         "margin_lo": -0.1, "frames": 1024, "iters": 20, "max_iter": 30},
        # a training step of that table: batch 512, 20 unrolled iterations
        {"name": "train_2_3_512", "kind": "train", "short": 0, "rate": "2_3", "const": "8PSK", "margin": 1.0,
         "margin_lo": 0.5, "frames": 512, "iters": 20},
        # the stages behind a decoded batch: most words clean, some corrected, a few beyond repair
        {"name": "outer_3_5_4096", "kind": "outer", "short": 0, "rate": "3_5", "frames": 4096, "corrected": 0.2,
         "lost": 0.05},
        # BCH parity of a transmit batch
        {"name": "encode_9_10_999", "kind": "encode", "short": 0, "rate": "9_10", "frames": 999},
        # the demapper in front of a decoded batch
        {"name": "demap_8psk_4096", "kind": "demap", "short": 0, "rate": "3_5", "const": "8PSK", "frames": 4096},
        # frames for training and testing
        {"name": "generate_8psk_1024", "kind": "generate", "short": 0, "rate": "2_3", "const": "8PSK",
         "margin": 0.5, "frames": 1024},
    ]


# committed learned tables: (short, rate, constellation, iterations)
LEARNED = [(s, r, "QPSK", 12) for s in (0, 1) for r in MC.RATES
           if not (s and r == "9_10")] + [(0, "2_3", "8PSK", 20), (0, "3_5", "8PSK", 30), (0, "3_5", "8PSK", 12)]
# constellations per frame size for the demapper, with a rate that has them
POINTS = [("QPSK", "1_2", 0), ("8PSK", "2_3", 0), ("16APSK", "3_4", 0), ("32APSK", "4_5", 0), ("QPSK", "1_3", 1),
          ("8PSK", "3_5", 1), ("16APSK", "5_6", 1), ("32APSK", "8_9", 1), ("64APSK", "128_180", 0),
          ("256APSK", "135_180", 0)]


def draw(rng):
    def spread(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["dropin", "decode", "decode", "host", "mixed", "learned", "train", "outer", "encode",
                       "demap", "generate"])
    if kind == "mixed":
        return {"kind": kind, "frames": spread(300, 2048), "max_iter": rng.choice([20, 30, 50])}
    if kind == "demap":
        const, rate, short = rng.choice(POINTS)
        most = 1024 if const in ("64APSK", "256APSK") else 4096
        return {"kind": kind, "short": short, "rate": rate, "const": const, "frames": spread(1, most)}
    short = int(rng.random() < 0.4)
    _, const, rate, _ = rng.choice([m for m in MC.MODCODS if not (short and m[2] == "9_10")])
    case = {"kind": kind, "short": short, "rate": rate}
    if kind == "outer":
        case.update(frames=spread(1, 4096), corrected=rng.choice([0.0, 0.05, 0.3, 1.0]), lost=0.0)
        if case["corrected"] < 1.0:
            case["lost"] = rng.choice([0.0, 0.05])
        return case
    if kind == "encode":
        case.update(frames=spread(1, 4096))
        return case
    case["const"] = const
    case["margin"] = round(rng.uniform(0.3, 1.2), 2)
    if kind == "generate":
        case.update(frames=spread(1, 2048))
        return case
    case["margin_lo"] = round(case["margin"] - rng.choice([0.0, 0.4, 1.0]), 2)
    if kind == "dropin":
        case.update(frames=rng.randint(1, 64), max_iter=rng.choice([20, 30, 50]))
    elif kind == "decode":
        case.update(frames=spread(1, 4096), max_iter=rng.choice([20, 30, 50]), stop=rng.choice([0, 0, 0, 32, 64]))
    elif kind == "host":
        case.update(frames=spread(64, 2048), max_iter=rng.choice([20, 30, 50]))
    elif kind == "learned":
        s, rate, const, iters = rng.choice(LEARNED)
        case.update(short=s, rate=rate, const=const, iters=iters, frames=spread(64, 2048), max_iter=30)
    else:
        # training keeps to frames that can be decoded
        lo = 1.0 if short else 0.5
        case.update(frames=spread(4, 256), iters=rng.randint(3, 20), margin=round(lo + rng.random(), 2), margin_lo=lo)
    return case


def qef(const, rate):
    try:
        return MC.qef_db(const, rate)
    except KeyError:  # a learned table's MODCOD outside the standard's list
        return min(q for c, q in MC.modcods_of_rate(rate, 0))


def frames_of(dec, case, seed):
    """A batch of the case's code on the GPU, Es/N0 in SPREAD points from
    margin_lo to margin: (LLRs int8 [n, N], information bits packed)."""
    n, base = case["frames"], qef(case["const"], case["rate"])
    llr = torch.empty((n, dec.N), dtype=torch.int8, device="cuda")
    info = torch.empty((n, dec.nbytes), dtype=torch.uint8, device="cuda")
    edges = [n * k // SPREAD for k in range(SPREAD + 1)]
    for k in range(SPREAD):
        a, b = edges[k], edges[k + 1]
        if b > a:
            es = base + case["margin_lo"] + (case["margin"] - case["margin_lo"]) * k / (SPREAD - 1)
            x, i, _ = dec.generate(b - a, es, seed=seed * 1000 + k, constellation=case["const"], info=True)
            llr[a:b], info[a:b] = x, i
    order = torch.randperm(n, generator=torch.Generator().manual_seed(seed)).cuda()
    return llr[order].contiguous(), info[order].contiguous()


def prepare(case, seed):
    kind, n = case["kind"], case["frames"]
    st = {"case": case}
    if kind == "mixed":
        return prepare_mixed(case, seed, st)
    if kind == "demap":
        st["demapper"] = D.Demapper(case["const"], case["rate"], case["short"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        # received symbols of unit mean power, one noise power per frame
        st["sym"] = torch.randn((n, 2 * st["demapper"].nsym), generator=g, device="cuda") * 0.7071
        st["n0"] = 10.0 ** (-(5.0 + 10.0 * torch.rand(n, generator=g, device="cuda")) / 10.0)
        st["llr"] = torch.empty((n, st["demapper"].nldpc), dtype=torch.int8, device="cuda")
        return st
    p = D.fec_lookup(case["short"], case["rate"])
    if kind in ("outer", "encode"):
        bch = st["bch"] = D.Bch(p)
        g = torch.Generator(device="cuda").manual_seed(seed)
        cw = torch.randint(0, 256, (n, bch.nbytes), generator=g, device="cuda", dtype=torch.uint8)
        st["cw"] = cw
        st["kbytes"] = p.kbch // 8
        if kind == "outer":
            bch.encode_device(cw)
            rng = np.random.default_rng(seed)
            kinds = rng.random(n)
            at, bit = [], []
            for f in np.nonzero(kinds < case["corrected"] + case["lost"])[0]:
                w = int(rng.integers(1, p.t + 1)) if kinds[f] < case["corrected"] else 300
                pos = rng.choice(p.kldpc, w, replace=False)
                at.append(f * bch.nbytes + pos // 8)
                bit.append(0x80 >> (pos % 8))
            if at:
                flips = np.zeros(n * bch.nbytes, np.uint8)
                np.bitwise_xor.at(flips, np.concatenate(at), np.concatenate(bit).astype(np.uint8))
                cw ^= torch.from_numpy(flips).cuda().view(n, bch.nbytes)
            st["received"] = cw.clone()
            st["result"] = torch.empty(n, dtype=torch.int32, device="cuda")
        return st
    if kind == "train":
        model = st["model"] = L.LearnedDecoder(case["short"], case["rate"], iters=case["iters"])
        beta, alpha = tables_of(case, seed, model.beta.shape[1])
        with torch.no_grad():
            model.beta.copy_(beta)
            model.alpha.copy_(alpha)
        llr, st["bits"] = frames_of(model.dec, case, seed)
        st["llr"] = llr.half()  # the int8 decoder's inputs, carried in FP16
        return st
    dec = st["dec"] = D.Ldpc(p, case["rate"])
    if kind == "generate":
        st["es"] = qef(case["const"], case["rate"]) + case["margin"]
        st["seed"] = seed * 1000
        return st
    llr, _ = frames_of(dec, case, seed)
    if kind == "dropin":
        st["llr"] = list(llr.cpu().numpy())
        st["out"] = np.zeros((n, dec.nbytes), np.uint8)
    elif kind == "host":
        def pinned(*shape, dtype):
            return torch.zeros(shape, dtype=dtype, pin_memory=True)
        st["keep"] = pinned(n, dec.N, dtype=torch.int8).copy_(llr)
        st["llr"] = st["keep"].numpy()
        st["out"] = pinned(n, dec.nbytes, dtype=torch.uint8).numpy()
        st["iters"] = pinned(n, dtype=torch.int32).numpy()
        st["ok"] = pinned(n, dtype=torch.uint8).numpy()
    else:
        st["llr"] = llr
        if kind == "learned":
            T.apply_table(dec, T.load_table(case["short"], case["rate"], case["const"], case["iters"]))
    return st


def prepare_mixed(case, seed, st):
    n = case["frames"]
    spec = MC.mixed_batch(n, seed=seed)
    codes = sorted(set((s, r) for s, r, _, _ in spec))
    at = {c: k for k, c in enumerate(codes)}
    code = np.array([at[(s, r)] for s, r, _, _ in spec], np.int32)
    decs = {c: D.Ldpc(D.fec_lookup(*c), c[1]) for c in codes}
    st["llr"] = torch.zeros((n, 64800), dtype=torch.int8, device="cuda")
    groups = {}
    for f, key in enumerate(spec):
        groups.setdefault(key, []).append(f)
    for g, ((s, r, const, es), rows) in enumerate(sorted(groups.items())):
        x, _, _ = decs[(s, r)].generate(len(rows), es, seed=seed * 1000 + g, constellation=const, const_rate=r)
        st["llr"][torch.tensor(rows, device="cuda"), : x.shape[1]] = x
    st["out"] = torch.zeros((n, max(d.nbytes for d in decs.values())), dtype=torch.uint8, device="cuda")
    st["iters"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    st["ok"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
    mix = st["mix"] = D.LdpcMix(codes)
    mix.plan(code, st["llr"], st["out"], st["iters"], st["ok"], case["max_iter"])
    mix.tune()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "dropin":
        it = st["dec"].decode(st["llr"], st["out"], case["max_iter"])
        return {"iterations": it, "bits": st["out"]}
    if kind == "decode":
        return st["dec"].decode_device(st["llr"], case["max_iter"], stop=case["stop"])
    if kind == "host":
        return st["dec"].decode_host(st["llr"], case["max_iter"], out=st["out"], iters=st["iters"], ok=st["ok"])
    if kind == "mixed":
        st["mix"].run()
        return st["out"], st["iters"], st["ok"]
    if kind == "learned":
        return st["dec"].decode_learned(st["llr"], case["iters"], plain_max_iter=case["max_iter"])
    if kind == "train":
        model = st["model"]
        model.zero_grad(set_to_none=True)
        loss = model(st["llr"], st["bits"])
        loss.backward()
        return {"loss": loss.detach(), "scale_grad": model.beta.grad, "offset_grad": model.alpha.grad}
    if kind == "outer":
        # the LDPC decoder leaves every batch's words in this buffer
        st["cw"].copy_(st["received"])
        res = st["bch"].decode_device(st["cw"], result=st["result"])
        D.bb_descramble(st["cw"], st["kbytes"])
        return {"result": res, "header": D.bbheader_check(st["cw"]), "frames": st["cw"]}
    if kind == "encode":
        return st["bch"].encode_device(st["cw"])
    if kind == "demap":
        return st["demapper"].run(st["sym"], st["n0"], llr=st["llr"])
    llr, info, _ = st["dec"].generate(case["frames"], st["es"], seed=st["seed"], constellation=case["const"],
                                      info=True)
    return llr, info


MEAN_ITERS = 12  # iterations of a frame at the margins used here, on average


def work(case):
    """Bytes: every input once, every output once.  Operations: per link and
    iteration a subtraction, an absolute value, two minimum updates, a sign
    and an addition (three times that for a training step, which also walks
    every iteration back); per symbol and point two multiply-adds."""
    kind, n = case["kind"], case["frames"]
    if kind == "mixed":
        info = [D.code_info(s, r) for s, r, _, _ in MC.mixed_batch(n, seed=1)]
        return {"bytes": sum(i.nldpc + i.kldpc // 8 + 5 for i in info),
                "flops": 6 * MEAN_ITERS * sum(i.edges for i in info)}
    info = D.code_info(case["short"], case["rate"])
    N, nb, E = info.nldpc, info.kldpc // 8, info.edges
    if kind in ("dropin", "decode", "host", "learned"):
        return {"bytes": n * (N + nb + 5), "flops": 6 * MEAN_ITERS * n * E}
    if kind == "train":
        return {"bytes": n * (2 * N + nb), "flops": 3 * 6 * case["iters"] * n * E}
    if kind == "outer":
        kb = D.fec_lookup(case["short"], case["rate"]).kbch // 8
        return {"bytes": n * (nb + kb + 5), "flops": 0}
    if kind == "encode":
        return {"bytes": n * nb, "flops": 0}
    bits = {"QPSK": 2, "8PSK": 3, "16APSK": 4, "32APSK": 5, "64APSK": 6, "256APSK": 8}[case["const"]]
    if kind == "demap":
        nsym = -(-N // bits)
        return {"bytes": n * (8 * nsym + N + 4), "flops": n * nsym * 4 * (1 << bits)}
    return {"bytes": n * (N + nb), "flops": n * (-(-N // bits)) * 4 * (1 << bits)}


# ---- 64-bit values of the training step -------------------------------------------------------


def tables_of(case, seed, nclass):
    """Scale and offset tables as training meets them: near the plain
    decoder's ones, exact in FP16."""
    g = torch.Generator().manual_seed(seed)
    beta = 0.9 + 0.2 * torch.rand((case["iters"], nclass), generator=g)
    alpha = 0.6 + 0.5 * torch.rand((case["iters"], nclass), generator=g)
    return beta.half().float().cuda(), alpha.half().float().cuda()


@functools.lru_cache(maxsize=None)
def checks_of(short, rate):
    """The code's checks from the standard's address tables, in the decoder's
    order cut into steps of checks that share no bit: per step the bits of
    every check (int64 [checks, links], N: no link)."""
    text = open(os.path.join(HERE, "..", "dvbrx_b200", "csrc", "codes_gen.h")).read()
    rates = text.split("cg_rates_short[]" if short else "cg_rates_normal[]")[1].split("};")[0]
    table = int(re.search(r'\{ "%s", (\d+) \}' % rate, rates).group(1))
    row = re.findall(r'\{ "\w+", (\d+), (\d+), \d+, (\w+), (\w+) \}', text.split("cg_tables[]")[1].split("};")[0])
    N, K, runs, addr = row[table]
    N, K = int(N), int(K)
    runs, addr = (np.array(re.search(r"%s\[\] = \{(.*?)\};" % a, text, re.S).group(1).replace("\n", " ").strip(" ,")
                           .split(","), dtype=np.int64) for a in (runs, addr))
    R, q = N - K, (N - K) // 360
    layer = [[] for _ in range(q)]
    g = pos = 0
    for deg, count in runs.reshape(-1, 2):
        for _ in range(count):
            for a in addr[pos:pos + deg]:
                layer[a % q].append((g, a // q))
            pos += deg
            g += 1
    steps, j = [], np.arange(360)
    width = 2 + max(len(e) for e in layer)
    for i in range(q):
        # links that two checks of the layer can share first, then the others, in table order
        many = [e for e in layer[i] if sum(e[0] == f[0] for f in layer[i]) > 1]
        ent = many + [e for e in layer[i] if e not in many]
        bits = np.full((360, width), N)
        bits[:, 0] = K + q * j + i
        bits[:, 1] = np.where(q * j + i > 0, K + q * j + i - 1, N)
        for k, (g, a) in enumerate(ent):
            bits[:, 2 + k] = 360 * g + (j - a) % 360
        last, level = {}, np.zeros(360, np.int64)
        for c in range(360):
            shared = bits[c, 2:2 + len(many)].tolist()
            level[c] = max([last.get(b, -1) + 1 for b in shared], default=0)
            last.update((b, level[c]) for b in shared)
        steps += [bits[level == v] for v in range(level.max() + 1)]
    return N, K, steps


def exact(case, seed):
    if case["kind"] != "train":
        return None
    short, rate, iters, n = case["short"], case["rate"], case["iters"], case["frames"]
    p = D.fec_lookup(short, rate)
    dec = D.Ldpc(p, rate)
    llr, packed = frames_of(dec, case, seed)
    N, K, steps = checks_of(short, rate)
    degs = sorted(set(int(d) for s in steps for d in (s < N).sum(axis=1)))
    beta, alpha = (t.double() for t in tables_of(case, seed, len(degs)))
    sched = []
    first = 0
    for s in steps:
        idx = torch.from_numpy(s).cuda()
        cls = torch.tensor([degs.index(int(d)) for d in (s < N).sum(axis=1)], device="cuda")
        sched.append((idx, (idx < N)[:, :, None], cls, slice(first, first + len(s))))
        first += len(s)
    shifts = torch.arange(7, -1, -1, device="cuda", dtype=torch.uint8)
    loss = torch.zeros((), dtype=torch.float64, device="cuda")
    gb, ga = torch.zeros_like(beta), torch.zeros_like(alpha)
    denom = float(iters) * n * p.kldpc
    for a in range(0, n, 512):
        bits = ((packed[a:a + 512, :, None] >> shifts) & 1).reshape(-1, 8 * dec.nbytes)[:, : p.kldpc]
        sb = (1.0 - 2.0 * bits.double()).t()
        m = sb.shape[1]
        P = torch.zeros((N + 1, m), dtype=torch.float64, device="cuda")
        P[:N] = llr[a:a + 512].t().double().clamp(-128, 127)
        M = torch.zeros((first, steps[0].shape[1], m), dtype=torch.float64, device="cuda")
        saved = []
        for t in range(iters):
            saved.append((P.clone(), M.clone()))
            walk(P, M, sched, beta[t], alpha[t], None)
            loss += torch.nn.functional.softplus(-sb * P[: p.kldpc] / 2).sum() / denom
        gP, gM = torch.zeros_like(P), torch.zeros_like(M)
        for t in range(iters - 1, -1, -1):
            P, M = saved.pop()
            raws = []
            walk(P, M, sched, beta[t], alpha[t], raws)
            gP[: p.kldpc] += -0.5 * sb * torch.sigmoid(-sb * P[: p.kldpc] / 2) / denom
            for s in range(len(sched) - 1, -1, -1):
                back(gP, gM, sched[s], raws[s], beta[t], alpha[t], gb[t], ga[t])
        del saved, raws
    return {"loss": loss, "scale_grad": gb, "offset_grad": ga}


def node(raw, valid, beta, alpha):
    """A check node: inputs clamped, each link's message from the minimum
    and the sign of the others."""
    x = raw.clamp(-128, 127)
    mag = torch.where(valid, x.abs(), torch.inf)
    m0, a0 = mag.min(dim=1, keepdim=True)
    m1, a1 = mag.scatter(1, a0, torch.inf).min(dim=1, keepdim=True)
    own = torch.arange(raw.shape[1], device="cuda")[None, :, None] == a0
    mu = torch.where(own, m1, m0)
    pre = beta[:, None, None] * mu.clamp(max=127) - alpha[:, None, None]
    neg = (x < 0) & valid
    sign = 1.0 - 2.0 * ((neg.sum(dim=1, keepdim=True) + neg) % 2)
    return x, mu, torch.where(own, a1, a0), pre, sign, sign * pre.clamp(min=0)


def walk(P, M, sched, beta, alpha, raws):
    """One iteration in place; the extrinsic inputs of every step kept."""
    for idx, valid, cls, rows in sched:
        raw = P[idx] - M[rows]
        if raws is not None:
            raws.append(raw)
        x, _, _, _, _, msg = node(raw, valid, beta[cls], alpha[cls])
        P[idx] = (x + msg).clamp(-128, 127)
        M[rows] = torch.where(valid, msg.clamp(-32, 31), 0.0)


def back(gP, gM, step, raw, beta, alpha, gb, ga):
    """The gradients of a step's outputs to its inputs, in place: clamps that
    hold pass none, the minimum's goes to the link that has it."""
    idx, valid, cls, rows = step
    x, mu, src, pre, sign, msg = node(raw, valid, beta[cls], alpha[cls])
    post = x + msg
    gpost = torch.where((post >= -128) & (post <= 127) & valid, gP[idx], 0.0)
    gmsg = gpost + torch.where((msg >= -32) & (msg <= 31) & valid, gM[rows], 0.0)
    gmag = torch.where(pre > 0, gmsg * sign, 0.0)
    gb.index_add_(0, cls, (gmag * mu.clamp(max=127)).sum(dim=(1, 2)))
    ga.index_add_(0, cls, -gmag.sum(dim=(1, 2)))
    gmu = torch.where(mu < 127, gmag * beta[cls][:, None, None], 0.0)
    gx = gpost.scatter_add(1, src, gmu * torch.where(x.gather(1, src) < 0, -1.0, 1.0))
    g = torch.where((raw >= -128) & (raw <= 127), gx, 0.0)
    gP[idx] = g
    gM[rows] = -g
