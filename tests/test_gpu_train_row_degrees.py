"""The training kernel's row update for every degree it has one for, 2 to 32: codes of one degree, and codes
that mix a degree with short rows and rows of the class's largest, against the model of
oracle/learned_ref.py (the APPs bit for bit in its FP32 emulation, loss and gradients within the FP32
accumulation tolerance of the other training tests)."""
import numpy as np
import pytest

from oracle import learned_ref
from test_gpu_train_degrees import _code
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("d", range(2, 33))
def test_degree(cuda, d, mixed):
    import torch
    degrees = (d, 2, 8 if d <= 8 else (16 if d <= 16 else 32)) if mixed else (d,)
    n, m, F, T = 130 + d % 4, 24, 3, 2
    code = _code(n, m, degrees, 1000 + d)
    rng = np.random.default_rng(d)
    bits = rng.integers(0, 2, size=(F, n)).astype(np.uint8)
    llr = np.trunc(np.clip(8.0 * ((2.0 * bits - 1.0) + 0.8 * rng.standard_normal((F, n))), -31, 31))
    kappa = np.full(F, 0.3)
    alpha = rng.uniform(0.6, 1.1, (T, 2)).astype(np.float32)
    beta = rng.uniform(-0.5, 1.5, (T, 2)).astype(np.float32)
    w = np.array([0.5, 1.0])
    l_ref, app_ref, ga_ref, gb_ref = learned_ref.forward_backward(code, llr, bits, kappa, alpha, beta, weights=w,
                                                                  forward_dtype=np.float32)
    f32 = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda()
    dec = Decoder(code, "OMS", nb_frames=1)
    loss, app = torch.zeros(1, device="cuda"), torch.zeros(F, n, device="cuda")
    ga, gb = torch.zeros(T, 2, device="cuda"), torch.zeros(T, 2, device="cuda")
    stash = torch.empty(dec.train_stash_bytes(F, T), dtype=torch.uint8, device="cuda")
    dec.train_step(f32(llr), f32(kappa), F, T, f32(alpha), f32(beta), loss, d_bits=torch.from_numpy(bits).cuda(),
                   d_grad_alpha=ga, d_grad_beta=gb, d_stash=stash, d_app=app, d_weights=f32(w))
    torch.cuda.synchronize()
    dec.close()
    assert np.array_equal(app.cpu().numpy().astype(np.float64), app_ref)
    assert float(loss.item()) == pytest.approx(l_ref, rel=1e-5)
    scale = max(np.abs(ga_ref).max(), np.abs(gb_ref).max())
    assert np.abs(ga.cpu().numpy() - ga_ref).max() <= 5e-4 * scale
    assert np.abs(gb.cpu().numpy() - gb_ref).max() <= 5e-4 * scale
