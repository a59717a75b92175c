"""XMS on the per-frame early stop of the QC register kernel (decoder path 5): its input is interleaved by
words, which the kernel reads frame by frame.  Decisions, counts and flags equal the oracle's."""
import numpy as np
import pytest

import llr_gen
from gpu_helpers import make_llr
from oracle import oracle
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import qc_regular

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("pack", ["AUTO", "F16X2"])
@pytest.mark.parametrize("z,words", [(8, 1), (16, 7), (64, 700), (256, 150)])
def test_interleaved_input(cuda, z, words, pack, host):
    import torch
    code, iters = qc_regular(z=z, mb=8, nb=16, wc=3, seed=7, name="xms_%d" % z), 9
    llr = make_llr("awgn", 4 * words * code.n, 81, sigma=llr_gen.sigma_for(3.0, 0.5))
    ref = oracle.decode(code, "XMS", llr, iters, early_stop=True, per_frame=True)
    dec = Decoder(code, "XMS", nb_frames=words, pack=pack, early_stop="frame")
    assert dec.info()["path"] == 5
    if host:
        out, its = np.zeros((4 * words, code.n), np.uint8), np.zeros(4 * words, np.int32)
        dec.decode_host_ex(llr, out, iters, iters_out=its)
    else:
        o = torch.zeros(4 * words, code.n, dtype=torch.uint8, device="cuda")
        i = torch.zeros(4 * words, dtype=torch.int32, device="cuda")
        dec.decode_device(torch.from_numpy(llr).cuda(), o, words, iters, d_iters=i, stream=torch.cuda.current_stream())
        torch.cuda.synchronize()
        out, its = o.cpu().numpy(), i.cpu().numpy()
    dec.close()
    assert np.array_equal(out, np.asarray(ref["hard"]).reshape(4 * words, code.n))
    assert np.array_equal(its, np.asarray(ref["iters"]).reshape(-1))
