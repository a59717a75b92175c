"""The long-code kernel's memory (LDPC_PACK_FRAME) follows the code's edges, not its widest level: one wide
level and a long tail of one-row levels, and the serial 64800-column table.  Decisions and counts of the
first equal the oracle's."""
import numpy as np
import pytest

import llr_gen
from gpu_helpers import make_llr
from oracle import oracle
from fast_ldpc_decoder_for_gpu_fixed_b200 import Decoder, load_table
from fast_ldpc_decoder_for_gpu_fixed_b200.codes import Code

pytestmark = pytest.mark.gpu


def _wide_and_tail(wide, tail, d):
    """A level of ``wide`` rows of 3 variables, then ``tail`` rows that all hold variable 0."""
    n = 3 * wide + 7
    rng = np.random.default_rng(5)
    rows = [np.arange(3 * r, 3 * r + 3) for r in range(wide)]
    rows += [np.concatenate([[0], 1 + rng.choice(n - 1, size=d - 1, replace=False)]) for _ in range(tail)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    return Code("wide_%d_tail_%d" % (wide, tail), n, ptr, np.concatenate(rows).astype(np.int32),
                np.zeros(len(rows), np.uint8))


def _created(code, words):
    """(decoder, device bytes it took)"""
    import torch
    Decoder(load_table("576x288"), "OMS", nb_frames=1).close()  # the context and the library are loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    dec = Decoder(code, "OMS", nb_frames=words, pack="FRAME")
    assert dec.info()["path"] == 3
    return dec, free - torch.cuda.mem_get_info()[0]


def _limit(code, dec):
    """Twice the edges' bytes: a message of two frames per edge and resident CTA, each row's share rounded up
    to 16 bytes, and 64 bytes an edge of tables; and 32 MB for the allocator's rounding."""
    slots = 148 * max(1, dec.info()["ctas_per_sm"])
    return 2 * (slots * 16 * code.m + slots * 2 * code.e + 64 * code.e) + (32 << 20)


def test_wide_level_and_tail(cuda):
    import torch
    code, words, iters = _wide_and_tail(400, 3000, 7), 3, 4
    dec, took = _created(code, words)
    assert took <= _limit(code, dec)
    llr = make_llr("awgn", 4 * words * code.n, 51, sigma=llr_gen.sigma_for(3.0, 0.5))
    ref = oracle.decode(code, "OMS", llr, iters, per_frame=True)
    out = torch.zeros(4 * words, code.n, dtype=torch.uint8, device="cuda")
    its = torch.zeros(4 * words, dtype=torch.int32, device="cuda")
    dec.decode_device(torch.from_numpy(llr).cuda(), out, words, iters, d_iters=its, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert dec.status() == 0
    dec.close()
    assert np.array_equal(out.cpu().numpy(), np.asarray(ref["hard"]).reshape(4 * words, code.n))
    assert np.array_equal(its.cpu().numpy(), np.full(4 * words, iters))


def test_serial_table(cuda):
    code = load_table("64800x32400")
    dec, took = _created(code, 1)
    limit = _limit(code, dec)
    dec.close()
    assert took <= limit
