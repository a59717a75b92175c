"""The training kernel's row-degree classes (6, 7, up to 8, 16 and 32) with four-wide and scalar
access (n a multiple of 4 or not, LLRs on a 16-byte boundary or not), against the model of
oracle/learned_ref.py: the APPs bit for bit (its FP32 emulation), loss and gradients within the
FP32 accumulation tolerance of the other training tests."""
import numpy as np
import pytest

from oracle import learned_ref
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import Code

pytestmark = pytest.mark.gpu


def _code(n, m, degrees, seed):
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.choice(n, size=degrees[r % len(degrees)], replace=False)) for r in range(m)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    return Code("train_n%d_s%d" % (n, seed), n, ptr, np.concatenate(rows).astype(np.int32),
                (np.arange(m) >= m // 2).astype(np.uint8))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n,m,degrees", [(120, 50, (6,)), (121, 40, (7,)), (160, 60, (2, 5, 8)), (203, 40, (9, 16, 3)),
                                         (200, 30, (17, 32, 4)), (1600, 300, (6,))])
def test_degrees(cuda, n, m, degrees, shift):
    import torch
    code, F, T = _code(n, m, degrees, n + m), 5, 3
    rng = np.random.default_rng(7)
    bits = rng.integers(0, 2, size=(F, n)).astype(np.uint8)
    llr = np.trunc(np.clip(8.0 * ((2.0 * bits - 1.0) + 0.9 * rng.standard_normal((F, n))), -31, 31))
    kappa = np.full(F, 0.3)
    alpha = rng.uniform(0.6, 1.1, (T, 2)).astype(np.float32)
    beta = rng.uniform(-0.5, 1.5, (T, 2)).astype(np.float32)
    w = np.array([0.5, 0.0, 1.0])
    l_ref, app_ref, ga_ref, gb_ref = learned_ref.forward_backward(code, llr, bits, kappa, alpha, beta, weights=w,
                                                                  forward_dtype=np.float32)
    # shift: the LLRs start off a 16-byte boundary
    d_llr = torch.zeros(F * n + shift, dtype=torch.float32, device="cuda")[shift:]
    d_llr.copy_(torch.from_numpy(llr.astype(np.float32)).reshape(-1))
    f32 = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda()
    dec = Decoder(code, "OMS", nb_frames=1)
    loss, app = torch.zeros(1, device="cuda"), torch.zeros(F, n, device="cuda")
    ga, gb = torch.zeros(T, 2, device="cuda"), torch.zeros(T, 2, device="cuda")
    stash = torch.empty(dec.train_stash_bytes(F, T), dtype=torch.uint8, device="cuda")
    dec.train_step(d_llr, f32(kappa), F, T, f32(alpha), f32(beta), loss, d_bits=torch.from_numpy(bits).cuda(),
                   d_grad_alpha=ga, d_grad_beta=gb, d_stash=stash, d_app=app, d_weights=f32(w))
    torch.cuda.synchronize()
    dec.close()
    assert np.array_equal(app.cpu().numpy().astype(np.float64), app_ref)
    assert float(loss.item()) == pytest.approx(l_ref, rel=1e-5)
    scale = max(np.abs(ga_ref).max(), np.abs(gb_ref).max())
    assert np.abs(ga.cpu().numpy() - ga_ref).max() <= 5e-4 * scale
    assert np.abs(gb.cpu().numpy() - gb_ref).max() <= 5e-4 * scale
