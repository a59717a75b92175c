"""The long-code kernel's stages (LDPC_PACK_FRAME) where they can go wrong: rows of one degree and of
many in a level (lists padded to 4, 8 and 14), both row classes, levels wider than a stage, so few
stages that one frame per CTA serves the code, five to nine stages (the copies' fences), and an odd
number of variables.  Decisions, per-frame counts and flags equal the oracle's exactly."""
import numpy as np
import pytest

import llr_gen
from gpu_helpers import make_llr
from oracle import oracle
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import Code

pytestmark = pytest.mark.gpu


def _layers(n, layers, rows, degrees, seed, classes=False):
    """``layers`` levels of ``rows`` rows (each level on its own permutation of the variables)."""
    rng = np.random.default_rng(seed)
    cols, deg, cls = [], [], []
    for l in range(layers):
        perm, at = rng.permutation(n), 0
        for r in range(rows):
            d = degrees[(l + r) % len(degrees)]
            cols.append(perm[at:at + d])
            at += d
            deg.append(d)
            cls.append((l + r) % 2 if classes else 0)
        assert at <= n
    return Code("layers_n%d_l%d_s%d" % (n, layers, seed), n, np.concatenate([[0], np.cumsum(deg)]).astype(np.int32),
                np.concatenate(cols).astype(np.int32), np.array(cls, dtype=np.uint8))


CODES = {
    "degree_6": (1200, 9, 200, (6,)),
    "two_degrees": (1201, 7, 150, (5, 6)),
    "mixed_4": (600, 8, 100, (1, 2, 3, 4)),
    "mixed_8": (900, 12, 100, (8, 3, 5, 7)),
    "mixed_14": (1600, 5, 90, (14, 9, 2, 11, 13)),
    "wide": (4096, 6, 1024, (4,)),
    "nine_stages": (400, 9, 50, (7,)),
    "five_stages": (400, 5, 50, (7,)),
    "three_stages": (400, 3, 50, (7,)),
}


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("kind", ["OMS", "NMS"])
@pytest.mark.parametrize("name", sorted(CODES))
def test_stages(cuda, name, kind, early):
    import torch
    code = _layers(*CODES[name], seed=len(name), classes=name in ("two_degrees", "mixed_8", "nine_stages"))
    words, iters = 3, 6
    llr = make_llr("awgn", 4 * words * code.n, 31, sigma=llr_gen.sigma_for(5.0, 0.5))
    llr[:code.n] = make_llr("extreme", code.n, 32)
    ref = oracle.decode(code, kind, llr, iters, early_stop=early, per_frame=True)
    dec = Decoder(code, kind, nb_frames=words, pack="FRAME", early_stop=early)
    assert dec.info()["path"] == 3
    out = torch.zeros(4 * words, code.n, dtype=torch.uint8, device="cuda")
    its = torch.zeros(4 * words, dtype=torch.int32, device="cuda")
    syn = torch.zeros(4 * words, dtype=torch.uint8, device="cuda")
    dec.decode_device(torch.from_numpy(llr).cuda(), out, words, iters, d_iters=its, d_syndrome=syn,
                      stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert dec.status() == 0
    dec.close()
    hard = np.asarray(ref["hard"]).reshape(4 * words, code.n)
    assert np.array_equal(out.cpu().numpy(), hard)
    assert np.array_equal(its.cpu().numpy(), np.asarray(ref["iters"]).reshape(-1) if early else np.full(4 * words, iters))
    odd = np.zeros((code.m, 4 * words), dtype=np.int64)
    np.add.at(odd, np.repeat(np.arange(code.m), np.diff(code.row_ptr)), hard[:, code.cols].T)
    assert np.array_equal(syn.cpu().numpy(), (odd % 2 == 0).all(axis=0).astype(np.uint8))
