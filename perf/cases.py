"""What a user of this framework has it do, as cases that can be timed.

`listed()` are fixed cases over the range of real use: one 4-frame word (latency), the tables of the
reference with one and two degree groups at their usual batch sizes, fixed iterations and early stop,
QC codes in the register kernels, a mixed batch of short irregular codes, a long code, the fused
Monte-Carlo step, the host call of the plugin classes, and a training step.  `draw(rng)` gives more
cases of the same ranges.

Every frame is the transmission the decoders are built for: BPSK over AWGN at an Eb/N0 near the code's
waterfall, quantised like the reference channel, q = trunc(clamp(8y, -31, 31)), bit 1 positive.
"""
import functools
import os

import numpy as np
import torch

import fast_ldpc_decoder_for_gpu_fixed_b200 as fl
from fast_ldpc_decoder_for_gpu_fixed_b200 import _lib, codes, learned

TRAINED = os.path.join(learned.TRAINED_DIR, "qc3x6_z256_T10_offsets.json")

# The reference's tables that decode with more than a handful of rows at a time or are short enough
# for a serial schedule to be useful (the two 64800-column tables are one row at a time).
TABLES = ("576x288", "816x408", "1024x518", "1200x600", "1944x972", "2048x384", "2304x1152", "4000x2000",
          "4896x2448", "8000x4000", "9972x4986")


def listed():
    return [
        # the smallest call: one word of a short table, as a receiver decodes it when it arrives
        {"name": "word_576", "call": "device", "code": "576x288", "kind": "OMS", "words": 1, "iters": 20, "ebn0": 2.5},
        # the reference's default run: its default table, OMS, 20 iterations, -n 1024
        {"name": "table_4000_oms", "call": "device", "code": "4000x2000", "kind": "OMS", "words": 1024, "iters": 20,
         "ebn0": 2.0},
        # two degree groups, an odd number of words, packed bits and the per-frame syndrome flags
        {"name": "table_1944_nms_packed", "call": "device", "code": "1944x972", "kind": "NMS", "words": 777,
         "iters": 30, "ebn0": 2.5, "packed": True, "syndrome": True},
        # the reference's own early termination, decided per 4-frame word
        {"name": "table_2304_2nms", "call": "device", "code": "2304x1152", "kind": "2NMS", "words": 1500, "iters": 20,
         "ebn0": 3.0},
        # a large table whose words stop at the first codeword: few words on the chip at a time
        {"name": "table_9972_early", "call": "device", "code": "9972x4986", "kind": "OMS", "words": 501, "iters": 50,
         "ebn0": 2.5, "early": "word"},
        # QC code with every message in registers, fixed iterations, 65 536 frames
        {"name": "qc256_oms", "call": "device", "code": "qc256", "kind": "OMS", "words": 16384, "iters": 10,
         "ebn0": 2.0},
        # the deployed learned-offset decoder on that code, each frame pair stopping on its own
        {"name": "qc256_learned_pairs", "call": "device", "code": "qc256", "kind": "LEARNED", "words": 16384,
         "iters": 10, "ebn0": 2.25, "early": "pairs", "slack": _lib.EARLY_SLACK_ANY},
        # short irregular codes of four rates in one launch, Zipf(1.2) shares of 200 000 frames, early stop
        {"name": "batch_irregular", "call": "batch", "kind": "OMS", "words": 50000, "iters": 20, "ebn0": 3.0,
         "early": "word", "z": 54, "per_code": False},
        # a broadcast-length code, at most 50 iterations, each frame stopping on its own
        {"name": "ira_64800_early", "call": "device", "code": "ira", "kind": "OMS", "words": 512, "iters": 50,
         "ebn0": 1.4, "early": "word"},
        # one step of a Monte-Carlo run: channel, decoder and error count in one call
        {"name": "simulate_4000", "call": "simulate", "code": "4000x2000", "kind": "OMS", "words": 2048, "iters": 20,
         "ebn0": 1.75},
        # the plugin classes' decode() between host buffers
        {"name": "host_4000_oms", "call": "host", "code": "4000x2000", "kind": "OMS", "words": 1024, "iters": 20,
         "ebn0": 2.0},
        # a training step of the learned constants: quantised forward pass, loss and gradients
        {"name": "train_qc256", "call": "train", "code": "qc256", "words": 512, "iters": 10, "ebn0": 2.0,
         "frame_loss": False},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["device", "device", "device", "device", "early", "early", "qc", "irregular", "batch", "long",
                       "simulate", "host", "train"])
    if call in ("device", "early"):
        case = {"call": "device", "code": rng.choice(TABLES), "iters": _log(rng, 2, 50)}
        n = int(case["code"].split("x")[0])
        rows = int(case["code"].split("x")[1])
        # the two tables with the longest serial schedules get fewer frames, as they are much slower
        most = min(20_000_000 // n, 400_000 // n if rows in (518, 600) else 1 << 30)
        case["words"] = _log(rng, 1, max(2, most // 4))
        case["ebn0"] = round(rng.uniform(1.5, 3.5), 2)
        if call == "early":
            case["early"] = rng.choice(["word", "frame"])
            case["kind"] = rng.choice(["MS", "OMS", "NMS"])
        else:
            case["kind"] = rng.choice(["MS", "OMS", "OMS", "NMS", "2NMS", "XMS"])
        case["packed"] = rng.random() < 0.3
        case["syndrome"] = rng.random() < 0.3
        return case
    if call == "qc":
        case = {"call": "device", "code": rng.choice(["qc64", "qc128", "qc256", "qc256"]), "iters": _log(rng, 5, 20),
                "words": _log(rng, 64, 12000), "ebn0": round(rng.uniform(1.75, 2.75), 2)}
        case["kind"] = rng.choice(["OMS", "NMS", "LEARNED"])
        if rng.random() < 0.6:
            case["early"] = rng.choice(["word", "pairs"])
            case["slack"] = rng.choice([_lib.EARLY_STOP_DEFAULT_SLACK, _lib.EARLY_SLACK_ANY])
        return case
    if call == "irregular":
        case = {"call": "device", "code": "irr%d_%s" % (rng.choice([27, 54, 81, 96]), rng.choice(["12", "23", "34", "56"])),
                "kind": rng.choice(["MS", "OMS", "NMS", "2NMS"]), "iters": _log(rng, 5, 30),
                "words": _log(rng, 1, 6000), "ebn0": round(rng.uniform(2.0, 3.5), 2)}
        if case["kind"] != "2NMS" and rng.random() < 0.5:
            case["early"] = rng.choice(["word", "frame"])
        return case
    if call == "batch":
        return {"call": "batch", "kind": rng.choice(["OMS", "NMS"]), "words": _log(rng, 100, 20000),
                "iters": _log(rng, 5, 20), "ebn0": round(rng.uniform(2.0, 4.0), 2),
                "early": rng.choice(["word", "frame", ""]), "z": rng.choice([27, 54, 81]),
                "per_code": rng.random() < 0.5}
    if call == "long":
        code = rng.choice(["ira", "ira", "20000x10000"])
        return {"call": "device", "code": code, "kind": rng.choice(["OMS", "NMS"]), "words": _log(rng, 8, 300),
                "iters": _log(rng, 10, 40), "ebn0": round(rng.uniform(0.9, 1.3) + (0.5 if code == "ira" else 0.0), 2),
                "early": rng.choice(["word", ""]), "packed": rng.random() < 0.3}
    if call == "simulate":
        return {"call": "simulate", "code": rng.choice(["1944x972", "2304x1152", "4000x2000", "8000x4000", "qc128"]),
                "kind": "OMS", "words": _log(rng, 64, 2000), "iters": _log(rng, 5, 20),
                "ebn0": round(rng.uniform(1.0, 1.75), 2)}
    if call == "host":
        return {"call": "host", "code": rng.choice(["576x288", "1944x972", "4000x2000", "8000x4000"]), "kind": "OMS",
                "words": _log(rng, 16, 1500), "iters": _log(rng, 5, 20), "ebn0": round(rng.uniform(1.5, 3.0), 2)}
    return {"call": "train", "code": rng.choice(["qc128", "qc256", "1944x972", "4000x2000"]),
            "words": _log(rng, 32, 512), "iters": _log(rng, 4, 10), "ebn0": round(rng.uniform(1.0, 3.0), 2),
            "frame_loss": rng.random() < 0.5}


RATES = {"12": (1, 2), "23": (2, 3), "34": (3, 4), "56": (5, 6)}


@functools.lru_cache(maxsize=None)
def _code(name):
    if name.startswith("qc"):
        return codes.qc_regular(z=int(name[2:]), mb=8, nb=16, wc=3, seed=2024, name="qc3x6_z" + name[2:])
    if name.startswith("irr"):
        z, rate = name[3:].split("_")
        return codes.qc_irregular(z=int(z), rate=RATES[rate], seed=1300 + int(z))
    return codes.ira() if name == "ira" else codes.load_table(name)


@functools.lru_cache(maxsize=None)
def _codewords(name):
    """Some codewords of random information bits; the all-zero one, as the reference sends, for the code whose
    encoder takes too long to set up."""
    c = _code(name)
    return np.zeros((1, c.n), dtype=np.uint8) if name == "20000x10000" else learned.random_codewords(c, 64, 17)


def _channel(name, frames, ebn0, seed):
    """(bits, int8 LLRs), [frames][n], on the GPU."""
    c = _code(name)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    cw = torch.from_numpy(_codewords(name)).cuda()
    bits = cw[(torch.arange(frames, device="cuda") + seed) % cw.shape[0]]
    sigma = (2.0 * (c.n_info / c.n) * 10.0 ** (ebn0 / 10.0)) ** -0.5
    llr = torch.empty(frames, c.n, dtype=torch.int8, device="cuda")
    for f0 in range(0, frames, 4096):
        b = bits[f0:f0 + 4096]
        y = torch.randn(b.shape, generator=gen, device="cuda") * sigma + (2.0 * b.float() - 1.0)
        llr[f0:f0 + 4096] = (8.0 * y).clamp_(-31, 31).trunc_().to(torch.int8)
    return bits, llr


def _counts(case, path):
    """Iteration counts a decode reports: one per word, or per frame where each frame stops on its own."""
    return case["words"] * (4 if case.get("early") == "frame" or path == 3 else 1)


def _early(case):
    e = case.get("early")
    return e if e in ("frame", "pairs") else bool(e)


def _batch_parts(case):
    names = ["irr%d_%s" % (z, r) for z, r in zip((case["z"], 27, 81, 54), ("12", "23", "34", "56"))]
    share = 1.0 / np.arange(1, 5) ** 1.2
    return names, [max(1, int(round(case["words"] * s))) for s in share[[2, 0, 3, 1]] / share.sum()]


def prepare(case, seed):
    call = case["call"]
    st = dict(case)
    if call == "batch":
        names, words = _batch_parts(case)
        cs = [_code(x) for x in names]
        st["batch"] = fl.Batch(cs, case["kind"], early_stop=_early(case), graph=True)
        if case["per_code"]:
            st["batch"].configure(per_code=True, pack="SIMD4")
        st["n_words"] = words
        st["llr"] = [_channel(x, 4 * w, case["ebn0"], seed + i)[1] for i, (x, w) in enumerate(zip(names, words))]
        st["out"] = [torch.empty(4 * w, c.n, dtype=torch.uint8, device="cuda") for w, c in zip(words, cs)]
        per = 4 if case["early"] == "frame" else 1
        st["its"] = [torch.empty(w * per, dtype=torch.int32, device="cuda") for w in words]
        st["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()
        return st
    c = _code(case["code"])
    frames = 4 * case["words"]
    if call == "host":
        fl.select_code(c)
        st["plugin"] = fl.PLUGINS[case["kind"]](case["words"], c.n, c.m, c.e)
        st["plugin"].initialize()
        st["llr"] = _channel(case["code"], frames, case["ebn0"], seed)[1].cpu().numpy()
        st["out"] = np.empty((frames, c.n), dtype=np.uint8)
        return st
    if call == "train":
        T = case["iters"]
        st["dec"] = fl.Decoder(c, "OMS", nb_frames=1)
        st["bits"], llr = _channel(case["code"], frames, case["ebn0"], seed)
        st["llr"] = llr.float()
        st["alpha"], st["beta"], st["kappa"], st["weights"] = _train_constants(case, c, "cuda")
        st["stash"] = torch.empty(st["dec"].train_stash_bytes(frames, T), dtype=torch.uint8, device="cuda")
        st["loss"] = torch.zeros(1, device="cuda")
        st["grad_alpha"], st["grad_beta"] = torch.zeros(T, 2, device="cuda"), torch.zeros(T, 2, device="cuda")
        return st
    st["dec"] = fl.Decoder(c, case["kind"], nb_frames=case["words"], early_stop=_early(case))
    if case["kind"] == "LEARNED":
        off, sc, _ = learned.load_constants(TRAINED)
        st["dec"].set_learned(off, sc)
    if case.get("slack"):
        st["dec"].set_early_stop(True, case["slack"])
    if call == "simulate":
        st["sigma"] = (2.0 * (c.n_info / c.n) * 10.0 ** (case["ebn0"] / 10.0)) ** -0.5
        st["seed"] = seed
        st["cw"] = torch.from_numpy(_codewords(case["code"])).cuda()
        st["counts"] = torch.zeros(3, dtype=torch.int64, device="cuda")
        return st
    st["llr"] = _channel(case["code"], frames, case["ebn0"], seed)[1]
    if case["kind"] == "XMS":  # that plugin reads word[v * words + g], byte k = frame 4g + k
        st["llr"] = st["llr"].view(case["words"], 4, c.n).permute(2, 0, 1).contiguous()
    st["format"] = _lib.OUT_PACKED if case.get("packed") else _lib.OUT_BYTES
    st["out"] = torch.empty(frames, (c.n + 7) // 8 if case.get("packed") else c.n, dtype=torch.uint8, device="cuda")
    st["its"] = torch.empty(_counts(case, st["dec"].info()["path"]), dtype=torch.int32, device="cuda")
    st["syn"] = torch.empty(frames, dtype=torch.uint8, device="cuda") if case.get("syndrome") else None
    return st


def run(st):
    call = st["call"]
    if call == "host":
        st["plugin"].decode(st["llr"], st["out"], st["iters"])
        return st["out"]
    if call == "batch":
        st["stream"].wait_stream(torch.cuda.current_stream())
        st["batch"].decode(st["llr"], st["out"], st["n_words"], st["iters"], d_iters=st["its"], stream=st["stream"])
        torch.cuda.current_stream().wait_stream(st["stream"])
        return [st["out"], st["its"]]
    stream = torch.cuda.current_stream()
    if call == "train":
        for k in ("loss", "grad_alpha", "grad_beta"):
            st[k].zero_()
        st["dec"].train_step(st["llr"], st["kappa"], 4 * st["words"], st["iters"], st["alpha"], st["beta"], st["loss"],
                             d_bits=st["bits"], quantized=True, d_grad_alpha=st["grad_alpha"],
                             d_grad_beta=st["grad_beta"], d_stash=st["stash"], d_weights=st["weights"],
                             frame_loss=st["frame_loss"], stream=stream)
        return {k: st[k] for k in ("loss", "grad_alpha", "grad_beta")}
    if call == "simulate":
        st["counts"].zero_()
        st["dec"].simulate(st["words"], st["iters"], st["sigma"], st["seed"], 0, st["counts"],
                           d_codewords=st["cw"], n_codewords=st["cw"].shape[0], stream=stream)
        return st["counts"]
    st["dec"].decode_device(st["llr"], st["out"], st["words"], st["iters"], out_format=st["format"], d_iters=st["its"],
                            stream=stream, d_syndrome=st["syn"])
    return [st["out"], st["its"]] + ([st["syn"]] if st["syn"] is not None else [])


# The iterations a decoder with early stop needs on average at these operating points, at the least.
STOPPED = {"ira": 20}


def work(case):
    if case["call"] == "batch":
        names, words = _batch_parts(case)
        parts = [(_code(x), 4 * w) for x, w in zip(names, words)]
    else:
        parts = [(_code(case["code"]), 4 * case["words"])]
    iters = case["iters"]
    if case.get("early") or case.get("kind") == "2NMS":
        iters = min(iters, STOPPED.get(case.get("code"), 5))
    if case["call"] == "train":  # float LLRs and bits in, the gradients out; forward and backward
        return {"bytes": sum(f * 5 * c.n for c, f in parts), "flops": sum(3 * 8 * f * c.e * iters for c, f in parts)}
    out = {"simulate": 0.0}.get(case["call"], 0.125 if case.get("packed") else 1.0)
    into = 0.0 if case["call"] == "simulate" else 1.0
    # 8 integer lane operations an edge and iteration: subtract, abs, two minima, sign, select, negate, add
    return {"bytes": int(sum(f * c.n * (into + out) for c, f in parts)), "flops": sum(8 * f * c.e * iters for c, f in parts)}


# ---- the training step in 64 bits ----------------------------------------------------------------


def _train_constants(case, c, device):
    """Constants on the grids of the quantised pass (scales s / 128 in steps of 8, integer offsets)."""
    T = case["iters"]
    t = torch.arange(T, dtype=torch.float32)
    alpha = torch.stack([(120 - 8 * (t % 3)) / 128, torch.full((T,), 1.0)], dim=1)
    beta = torch.stack([1.0 - (t % 2), torch.ones(T)], dim=1)
    sigma2 = 1.0 / (2.0 * (c.n_info / c.n) * 10.0 ** (case["ebn0"] / 10.0))
    kappa = torch.full((4 * case["words"],), 1.0 / (4.0 * sigma2))
    weights = torch.full((T,), 1.0 / T)
    return tuple(x.contiguous().to(device) for x in (alpha, beta, kappa, weights))


def _levels(c):
    """Rows that share no variable with an earlier row of their group, in order: [(columns [rows][d], group)]."""
    last = np.full(c.n, -1)
    at = {}
    for r in range(c.m):
        cols = c.cols[c.row_ptr[r]:c.row_ptr[r + 1]]
        lv = last[cols].max() + 1
        last[cols] = lv
        at.setdefault((lv, len(cols), int(c.row_class[r])), []).append(cols)
    return [(torch.tensor(np.array(v)).long(), k[2]) for k, v in sorted(at.items())]


def exact(case, seed):
    if case["call"] != "train":
        return None  # decisions, counts and flags are whole numbers
    c = _code(case["code"])
    bits, llr = _channel(case["code"], 4 * case["words"], case["ebn0"], seed)
    alpha, beta, kappa, weights = (x.double() for x in _train_constants(case, c, "cuda"))
    groups = [(cols.cuda(), g) for cols, g in _levels(c)]
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    d_alpha, d_beta = torch.zeros_like(alpha), torch.zeros_like(beta)
    F = llr.shape[0]
    part = max(1, min(F, (1 << 28) // (c.e * case["iters"])))  # frames at a time
    for f0 in range(0, F, part):
        s = slice(f0, f0 + part)
        _train_part(c.n, F, groups, llr[s].double(), bits[s].double(), kappa[s], alpha, beta, weights,
                    case["frame_loss"], loss, d_alpha, d_beta)
    return {"loss": loss, "grad_alpha": d_alpha, "grad_beta": d_beta}


def _train_part(n, F, groups, a, bits, kappa, alpha, beta, weights, frame_loss, loss, d_alpha, d_beta):
    kap = kappa[:, None]
    msg = [torch.zeros((), dtype=torch.float64, device="cuda")] * len(groups)
    keep, apps = [], []
    for t in range(alpha.shape[0]):
        rows = []
        for i, (cols, g) in enumerate(groups):
            tv = (a[:, cols] - msg[i]).clamp(-128, 127)
            pos = tv > 0
            mags, order = tv.abs().clamp(max=127).sort(dim=2, stable=True)
            mins, arg = mags[..., :2].clone(), order[..., :2].clone()
            odd = pos.sum(2, keepdim=True) % 2 == 1
            mag = (torch.floor(alpha[t, g] * mins) - beta[t, g])
            c1, c2 = mag[..., 1:].clamp(0, 31), mag[..., :1].clamp(0, 31)
            sign = torch.where(odd ^ pos, 1.0, -1.0).double()
            msg[i] = sign * torch.where(torch.arange(cols.shape[1], device="cuda") == arg[..., :1], c1, c2)
            a[:, cols] = (tv + msg[i]).clamp(-128, 127)
            rows.append((mins, arg.to(torch.int8), sign.to(torch.int8), pos))
        keep.append(rows)
        z = kap * a
        S = (z.clamp(min=0) + torch.log1p(torch.exp(-z.abs())) - bits * z).sum(1)
        loss += weights[t] * ((1 - torch.exp(-S)).sum() / F if frame_loss else S.sum() / (F * n))
        factor = torch.exp(-S)[:, None] / F if frame_loss else 1.0 / (F * n)
        apps.append(weights[t] * factor * kap * (torch.sigmoid(z) - bits))
    ga = torch.zeros_like(a)
    gmsg = [torch.zeros((), dtype=torch.float64, device="cuda")] * len(groups)
    for t in range(alpha.shape[0] - 1, -1, -1):
        ga += apps[t]
        for i in range(len(groups) - 1, -1, -1):
            cols, g = groups[i]
            mins, arg, sign, pos = keep[t][i]
            arg = arg.long()
            gt = ga[:, cols]
            sg = sign.double() * (gt + gmsg[i])
            first = sg.gather(2, arg[..., :1])
            gc = torch.cat([sg.sum(2, keepdim=True) - first, first], dim=2)  # by the smallest, by the second
            y = torch.floor(alpha[t, g] * mins) - beta[t, g]
            gc = gc * ((y > 0) & (y < 31))
            d_alpha[t, g] += (mins * gc).sum()
            d_beta[t, g] -= gc.sum()
            up = torch.where(pos.gather(2, arg), 1.0, -1.0).double()
            gt = gt.scatter_add(2, arg, up * alpha[t, g] * gc)
            ga[:, cols] = gt
            gmsg[i] = -gt
