"""LDPC_LEARNED on QC register kernels whose CTA has fewer threads than there are constants: as many
iterations of constants as a decoder holds, on lifting sizes below 64.  Decisions, counts equal the
oracle's exactly."""
import numpy as np
import pytest

import llr_gen
from gpu_helpers import make_llr
from oracle import oracle
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder, _lib
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import qc_irregular, qc_regular

pytestmark = pytest.mark.gpu

ITERS = 32  # LDPC_LEARNED_MAX_ITERS


def _constants(offsets_only):
    t = np.arange(ITERS)
    off = np.stack([t % 3, (t + 1) % 2], axis=1).astype(np.int8)
    sc = np.full((ITERS, 2), 128) if offsets_only else np.stack([128 - 8 * (t % 4), 120 + 0 * t], axis=1)
    return off, sc.astype(np.uint8)


CASES = [("regular", z, "AUTO", e, s) for z in (8, 16, 32, 64) for e, s in
         ((False, None), (True, 64), ("pairs", 64), ("pairs", _lib.EARLY_SLACK_ANY), ("frame", 64))]
CASES += [("irregular", z, pack, e, 64 if e else None) for z in (27, 54) for pack in ("F16X2", "F16X2_SPLIT") for e in (False, True)]


@pytest.mark.parametrize("offsets_only", [False, True])
@pytest.mark.parametrize("base,z,pack,early,slack", CASES)
def test_small_lifting(cuda, base, z, pack, early, slack, offsets_only):
    import torch
    code = qc_regular(z=z, mb=8, nb=16, wc=3, seed=7, name="small_%d" % z) if base == "regular" else \
        qc_irregular(z=z, rate=(1, 2), seed=9)
    off, sc = _constants(offsets_only)
    oracle.set_learned(off, sc)
    words = 4
    llr = make_llr("awgn", 4 * words * code.n, 71 + z, sigma=llr_gen.sigma_for(1.5, 0.5))
    half = pack != "AUTO"  # 2 frames per CTA: the stop is per frame pair
    ref = oracle.decode(code, "LEARNED", llr, ITERS, early_stop=bool(early), early_slack=slack or 0, per_frame=early == "frame",
                        pairs=early == "pairs" or (half and bool(early)))
    dec = Decoder(code, "LEARNED", nb_frames=words, pack=pack, early_stop=early)
    assert dec.info()["path"] == ({"frame": 5}.get(early, 1) if base == "regular" else (7 if pack == "F16X2_SPLIT" else 4))
    dec.set_learned(off, sc)
    if early:
        dec.set_early_stop(True, slack)
    out = torch.zeros(4 * words, code.n, dtype=torch.uint8, device="cuda")
    its = torch.zeros(4 * words if early == "frame" else words, dtype=torch.int32, device="cuda")
    dec.decode_device(torch.from_numpy(llr).cuda(), out, words, ITERS, d_iters=its, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    dec.close()
    assert np.array_equal(out.cpu().numpy(), np.asarray(ref["hard"]).reshape(4 * words, code.n))
    assert np.array_equal(its.cpu().numpy(), np.asarray(ref["iters"]).reshape(-1))
