"""The error counts of ldpc_simulate against its own decisions, where the counting can go wrong: CTAs whose
last warp is not full (QC kernels with a lifting size that is no multiple of 32), and the two frames of a
long-code CTA, which are counted one right after the other."""
import numpy as np
import pytest

from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder, load_table
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import qc_irregular, qc_regular

pytestmark = pytest.mark.gpu


def _counts(code, words, iters, sigma, n_vars, **kw):
    """(path, counts of the decoder, the same from its decisions); the all-zero codeword is sent."""
    import torch
    dec = Decoder(code, "OMS", nb_frames=words, **kw)
    counts = torch.zeros(3, dtype=torch.int64, device="cuda")
    hard = torch.zeros(4 * words, code.n, dtype=torch.uint8, device="cuda")
    dec.simulate(words, iters, sigma, 91, 3, counts, n_vars=n_vars, d_hard=hard, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    path = dec.info()["path"]
    dec.close()
    bits = hard.cpu().numpy()[:, :n_vars].sum(axis=1, dtype=np.int64)
    return path, counts.cpu().numpy().tolist(), [4 * words, int(bits.sum()), int((bits != 0).sum())]


@pytest.mark.parametrize("n_vars", [1, 40, 150])
@pytest.mark.parametrize("base,z,pack", [("irregular", 27, "F16X2"), ("irregular", 54, "F16X2"), ("irregular", 81, "F16X2"),
                                         ("irregular", 27, "F16X2_SPLIT"), ("irregular", 54, "F16X2_SPLIT"),
                                         ("regular", 16, "AUTO"), ("regular", 64, "AUTO"), ("irregular", 27, "SIMD4")])
def test_last_warp_not_full(cuda, base, z, pack, n_vars):
    code = qc_regular(z=z, mb=8, nb=16, wc=3, seed=7, name="small_%d" % z) if base == "regular" else \
        qc_irregular(z=z, rate=(1, 2), seed=9)
    path, got, want = _counts(code, 40, 2, 1.1, n_vars, pack=pack)
    assert path == (1 if base == "regular" else {"F16X2": 4, "F16X2_SPLIT": 7, "SIMD4": 0}[pack])
    assert got == want and want[1] > 0


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("n_vars", [0, 1, 33, 576])
@pytest.mark.parametrize("name", ["576x288", "1944x972"])
def test_two_frames_of_a_cta(cuda, name, n_vars, early):
    path, got, want = _counts(load_table(name), 300, 3, 0.9, n_vars, pack="FRAME", early_stop=early)
    assert path == 3
    assert got == want
