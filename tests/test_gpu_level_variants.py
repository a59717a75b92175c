"""Which level kernel a decoder runs (ldpc_decoder_level_info), and that each variant of the one with byte
storage gives the oracle's result: rows of 6 and 7 edges everywhere and of any number, two frame pairs and
one a thread, one a CTA, without the early stop, with it per word and per frame."""
import numpy as np
import pytest

import llr_gen
from gpu_helpers import make_llr
from oracle import oracle
from test_gpu_level_bytes import CODES
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder

pytestmark = pytest.mark.gpu

DEGREES = {"6": "576x288", "7": "one_level", "any": "irregular"}
MANY, FEW = 6000, 2  # words of a decoder that the chip is filled with, and not


@pytest.mark.parametrize("pack", ["SIMD4", "F16X2"])
@pytest.mark.parametrize("name", sorted(CODES))
def test_byte_kernel_serves(cuda, name, pack):
    """Every code but those with a repeated variable in a row or more variables than the records hold."""
    dec = Decoder(CODES[name](), "OMS", nb_frames=3, pack=pack)
    info, path = dec.level_info(), dec.info()["path"]
    dec.close()
    assert path == (0 if pack == "SIMD4" else 2)
    assert info["bytes"] == (name not in ("repeated", "n_16385"))
    assert (info["steps"] > 0) == (info["pairs_per_thread"] > 0) == bool(info["bytes"])


def _decoded(code, kind, pack, early, nb_frames):
    """Decodes FEW words, compares with the oracle; returns the variant that ran."""
    import torch
    words, iters = FEW, 8
    llr = make_llr("awgn", 4 * words * code.n, 61, sigma=llr_gen.sigma_for(4.0, 0.5))
    llr[:code.n] = make_llr("extreme", code.n, 62)
    ref = oracle.decode(code, kind, llr, iters, early_stop=bool(early), per_frame=early == "frame")
    dec = Decoder(code, kind, nb_frames=nb_frames, pack=pack, early_stop=early)
    out = torch.zeros(4 * words, code.n, dtype=torch.uint8, device="cuda")
    its = torch.zeros(4 * words if early == "frame" else words, dtype=torch.int32, device="cuda")
    dec.decode_device(torch.from_numpy(llr).cuda(), out, words, iters, d_iters=its, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    info = dec.level_info()
    dec.close()
    assert info["bytes"] == 1
    assert np.array_equal(out.cpu().numpy(), np.asarray(ref["hard"]).reshape(4 * words, code.n))
    assert np.array_equal(its.cpu().numpy(), np.asarray(ref["iters"]).reshape(-1))
    return "pair per CTA" if info["pair_per_cta"] else info["pairs_per_thread"]


@pytest.mark.parametrize("kind", ["MS", "OMS", "NMS"])
@pytest.mark.parametrize("early", [False, True, "frame"])
@pytest.mark.parametrize("degree", sorted(DEGREES))
def test_every_variant_runs(cuda, degree, early, kind):
    code = CODES[DEGREES[degree]]()
    ran = {_decoded(code, kind, "SIMD4", early, nb) for nb in (FEW, MANY)}
    if not early:
        ran |= {_decoded(code, kind, "F16X2", early, nb) for nb in (FEW, MANY)}
    assert ran == {1, 2} | (set() if early else {"pair per CTA"})


@pytest.mark.parametrize("degree", sorted(DEGREES))
def test_2nms_variants(cuda, degree):
    code = CODES[DEGREES[degree]]()
    assert {_decoded(code, "2NMS", "SIMD4", False, nb) for nb in (FEW, MANY)} == {1, 2}
