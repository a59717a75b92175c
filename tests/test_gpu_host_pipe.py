"""Host decode calls between pageable buffers (staged in pinned pieces, decisions expanded from packed
bits by host threads): bytes and packed bits, counts and flags equal the device call's on the
same LLRs, over one and several chunks and pieces, a number of variables that is not a multiple
of 8, and the decoder paths whose launches may and may not overlap; buffers below the staging's
size and pinned buffers take the direct copies."""
import numpy as np
import pytest

from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder, _lib, load_table
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import Code, ira, qc_regular

pytestmark = pytest.mark.gpu


def _odd():
    rng = np.random.default_rng(5)
    n, m = 1021, 300
    cols = np.concatenate([rng.choice(n, size=6, replace=False) for _ in range(m)])
    return Code("host_odd", n, (6 * np.arange(m + 1)).astype(np.int32), cols.astype(np.int32))


CASES = {"one_chunk": (lambda: load_table("4000x2000"), 66, {}), "many_pieces": (lambda: load_table("4000x2000"), 700, {}),
         "odd_n": (_odd, 530, {}), "small": (lambda: load_table("576x288"), 5, {}),
         "early_frames": (lambda: load_table("1944x972"), 401, {"early_stop": "frame"}),
         "frame_path": (lambda: ira(), 9, {"early_stop": True}),
         "qc_pairs": (lambda: qc_regular(z=64, mb=8, nb=16, wc=3, seed=5), 1100, {"early_stop": "pairs"})}


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_host_equals_device(cuda, name, pinned):
    import torch
    make, words, kw = CASES[name]
    code = make()
    dec = Decoder(code, "OMS", nb_frames=words, **kw)
    per = 4 if dec.info()["path"] in (3, 5) or kw.get("early_stop") == "frame" else 1
    rng = np.random.default_rng(7)
    host = lambda *shape, dtype: torch.zeros(*shape, dtype=dtype, pin_memory=True).numpy() if pinned else \
        np.zeros(shape, dtype={torch.int8: np.int8, torch.uint8: np.uint8, torch.int32: np.int32}[dtype])
    llr = host(4 * words, code.n, dtype=torch.int8)
    out = host(4 * words, code.n, dtype=torch.uint8)
    packed = host(4 * words, (code.n + 7) // 8, dtype=torch.uint8)
    its, syn = np.zeros(words * per, np.int32), np.zeros(4 * words, np.uint8)
    for _ in range(2):  # new inputs through the same decoder
        llr[:] = np.clip(np.rint(rng.normal(-4, 5, size=llr.shape)), -31, 31)
        want = torch.zeros(4 * words, code.n, dtype=torch.uint8, device="cuda")
        d_its = torch.zeros(words * per, dtype=torch.int32, device="cuda")
        d_syn = torch.zeros(4 * words, dtype=torch.uint8, device="cuda")
        dec.decode_device(torch.from_numpy(llr).cuda(), want, words, 6, d_iters=d_its, d_syndrome=d_syn,
                          stream=torch.cuda.current_stream())
        torch.cuda.synchronize()
        want = want.cpu().numpy()
        out[:] = 9
        packed[:] = 9
        dec.decode_host_ex(llr, out, 6, iters_out=its, syndrome_ok=syn)
        dec.decode_host_ex(llr, packed, 6, out_format=_lib.OUT_PACKED)
        assert np.array_equal(out, want)
        assert np.array_equal(its, d_its.cpu().numpy()) and np.array_equal(syn, d_syn.cpu().numpy())
        assert np.array_equal(np.unpackbits(packed, axis=1, bitorder="little")[:, :code.n], want)
        out[:] = 9
        dec.decode_host(llr, out, 6)
        assert np.array_equal(out, want)
    dec.close()
