"""The level kernel with byte storage (decoder paths 0 and 2) at the edges of its schedule: two, one
and half the frame pairs of a word per thread and CTA (many and few words per decoder), rows over 1, 2 and 4 lanes, steps
cut within a level, rows that repeat a variable (the older level kernel) and more variables than
its 16-bit records hold.  Decisions, APP, messages and counts equal the oracle's exactly."""
import numpy as np
import pytest

import llr_gen
from gpu_helpers import make_llr
from oracle import oracle
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder, load_table
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import Code, qc_irregular

pytestmark = pytest.mark.gpu


def random_code(n, m, degrees, seed, repeat=False):
    """Rows of the given degrees (cycled) on random distinct variables; ``repeat``: one row holds a
    variable twice."""
    rng = np.random.default_rng(seed)
    rows = [rng.choice(n, size=degrees[r % len(degrees)], replace=False) for r in range(m)]
    if repeat:
        rows[m // 2][-1] = rows[m // 2][0]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    cls = (np.arange(m) >= m // 2).astype(np.uint8)
    return Code("rnd_n%d_m%d_s%d%s" % (n, m, seed, "_rep" if repeat else ""), n, ptr,
                np.concatenate(rows).astype(np.int32), cls)


CODES = {
    "576x288": lambda: load_table("576x288"),
    "816x408": lambda: load_table("816x408"),        # degree 10: two lanes a row
    "2048x384": lambda: load_table("2048x384"),      # degree 32: four lanes of eight edges
    "9972x4986": lambda: load_table("9972x4986"),    # degree 7, levels wider than the CTA
    "irregular": lambda: _plain(qc_irregular(z=27, rate=(3, 4), seed=300)),
    "degrees_1_to_19": lambda: random_code(301, 120, (1, 2, 3, 5, 8, 9, 13, 16, 17, 19), 1),
    "odd_n": lambda: random_code(1021, 90, (6,), 2),
    "one_level": lambda: _one_level(700, 100, 7),
    "repeated": lambda: random_code(203, 60, (5, 6), 3, repeat=True),
    "n_16385": lambda: random_code(16385, 300, (6,), 4),
}


def _plain(code):
    code.no_qc = True
    return code


def _one_level(n, m, d):
    """Every row on its own variables: one level, as wide as the code."""
    cols = np.arange(m * d, dtype=np.int32)
    return Code("one_level", n, (np.arange(m + 1) * d).astype(np.int32), cols, np.zeros(m, np.uint8))


@pytest.mark.parametrize("nb_frames", [3, 6000])
@pytest.mark.parametrize("kind,pack", [("OMS", "SIMD4"), ("2NMS", "SIMD4"), ("NMS", "SIMD4"), ("OMS", "F16X2"), ("MS", "F16X2")])
@pytest.mark.parametrize("name", sorted(CODES))
def test_state_matches_oracle(cuda, name, kind, pack, nb_frames):
    import torch
    code, words, iters = CODES[name](), 3, 5
    llr = make_llr("awgn", 4 * words * code.n, 11, sigma=llr_gen.sigma_for(2.0, 0.5))
    llr[:code.n] = make_llr("extreme", code.n, 12)
    ref = oracle.decode(code, kind, llr, iters, want_state=True)
    dec = Decoder(code, kind, nb_frames=nb_frames, pack=pack)
    d_llr = torch.from_numpy(llr).cuda()
    hard = torch.zeros(4 * words * code.n, dtype=torch.uint8, device="cuda")
    its = torch.zeros(words, dtype=torch.int32, device="cuda")
    app = torch.zeros(4 * words * code.n, dtype=torch.int8, device="cuda")
    msg = torch.zeros(4 * words * code.e, dtype=torch.int8, device="cuda")
    dec.decode_device_state(d_llr, hard, words, iters, its, app, msg, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    dec.close()
    for got, want in ((hard, ref["hard"]), (its, ref["iters"]), (app, ref["app"]), (msg, ref["msg"])):
        assert np.array_equal(got.cpu().numpy().reshape(-1), np.asarray(want).reshape(-1).astype(got.cpu().numpy().dtype))


@pytest.mark.parametrize("nb_frames", [2, 6000])
@pytest.mark.parametrize("early", [True, "frame"])
@pytest.mark.parametrize("name", ["576x288", "816x408", "irregular", "degrees_1_to_19"])
def test_early_stop_matches_oracle(cuda, name, early, nb_frames):
    import torch
    code, words, iters = CODES[name](), 2, 12
    llr = make_llr("awgn", 4 * words * code.n, 21, sigma=llr_gen.sigma_for(3.5, 0.5))
    ref = oracle.decode(code, "OMS", llr, iters, early_stop=True, per_frame=early == "frame")
    dec = Decoder(code, "OMS", nb_frames=nb_frames, early_stop=early)
    assert dec.info()["path"] == 0
    out = torch.zeros(4 * words, (code.n + 7) // 8, dtype=torch.uint8, device="cuda")
    its = torch.zeros(words * (4 if early == "frame" else 1), dtype=torch.int32, device="cuda")
    syn = torch.zeros(4 * words, dtype=torch.uint8, device="cuda")
    dec.decode_device(torch.from_numpy(llr).cuda(), out, words, iters, out_format=1, d_iters=its, d_syndrome=syn,
                      stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    dec.close()
    hard = np.unpackbits(out.cpu().numpy(), axis=1, bitorder="little")[:, :code.n]
    want = np.asarray(ref["hard"]).reshape(4 * words, code.n)
    assert np.array_equal(hard, want)
    assert np.array_equal(its.cpu().numpy(), np.asarray(ref["iters"]).reshape(-1))
    rows = np.repeat(np.arange(code.m), np.diff(code.row_ptr))
    odd = np.zeros((code.m, 4 * words), dtype=np.int64)
    np.add.at(odd, rows, want[:, code.cols].T)
    assert np.array_equal(syn.cpu().numpy(), (odd % 2 == 0).all(axis=0).astype(np.uint8))
