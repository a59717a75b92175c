"""Batch.set_early_stop after each way a batch can be set up: the persistent kernel, per-code launches
(configure, set_code_kernel) and what the autotuner leaves.  After the early stop is switched on, its slack
changed and switched off again, decisions and counts equal the oracle's under that rule, which is what a
batch created that way gives."""
import numpy as np
import pytest

from gpu_helpers import make_llr
from oracle import oracle
from test_gpu_batch import _check, _inputs, codes
from fast_ldpc_decoder_for_gpu_fixed_b200 import Batch, LdpcError, _lib

pytestmark = pytest.mark.gpu

SETUPS = ["persistent", "persistent_i8", "per_code", "set_code_kernel", "autotune", "back_to_persistent"]


def _setup(b, setup, args):
    if setup == "persistent_i8":
        b.configure(pack="I8", threads=96)
    elif setup == "per_code":
        b.configure(per_code=True, pack="SIMD4")
    elif setup == "set_code_kernel":
        b.set_code_kernel_one(1, 1)
    elif setup == "autotune":
        llrs, outs, words, its = args
        b.autotune(llrs, outs, words, 20, d_iters=its)
    elif setup == "back_to_persistent":
        b.configure(per_code=True, pack="F16X2")
        b.configure(threads=64, ctas_per_sm=2)


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("setup", SETUPS)
def test_toggled(cuda, setup, early):
    cs, words = codes(), [3, 1, 5, 2]
    host, llrs, outs, its = _inputs(cs, words, 41)
    b = Batch(cs, "OMS", early_stop=early)
    _setup(b, setup, (llrs, outs, words, its))
    before = b.info()
    for on, slack in ((not early, None), (True, 3), (True, None), (False, None), (early, None)):
        b.set_early_stop(on, _lib.EARLY_STOP_DEFAULT_SLACK if slack is None else slack)
        info = b.info()
        for key in ("pack", "threads", "per_code"):
            assert info[key] == before[key]
        for o, it in zip(outs, its):
            o.zero_()
            it.zero_()
        b.decode(llrs, outs, words, 20, d_iters=its)
        if slack is None:
            _check(cs, words, host, outs, its, "OMS", 20, on, batch=b)
        else:
            import torch
            torch.cuda.synchronize()
            for i, (c, w, llr, o, it) in enumerate(zip(cs, words, host, outs, its)):
                if b.info()["per_code"] and (b.code_info(i)["candidate"] == "FLOODING" or b.code_info(i)["path"] in (4, 7)):
                    continue  # another schedule or unit of the stop: checked above without the slack
                ref = oracle.decode(c, "OMS", llr, 20, interleaved=False, early_stop=True, early_slack=slack)
                assert np.array_equal(o.cpu().numpy().reshape(4 * w, c.n), ref["hard"])
                assert np.array_equal(it.cpu().numpy(), ref["iters"])
    b.close()


@pytest.mark.parametrize("setup", ["persistent", "per_code"])
def test_slack_of_the_per_frame_stop(cuda, setup):
    import torch
    cs, words = codes()[:2], [2, 3]
    host, llrs, outs, _ = _inputs(cs, words, 43)
    its = [torch.zeros(4 * w, dtype=torch.int32, device="cuda") for w in words]
    b = Batch(cs, "OMS", early_stop="frame")
    _setup(b, setup, None)
    b.set_early_stop(True, 2)
    b.decode(llrs, outs, words, 20, d_iters=its)
    torch.cuda.synchronize()
    for c, w, llr, o, it in zip(cs, words, host, outs, its):
        ref = oracle.decode(c, "OMS", llr, 20, interleaved=False, early_stop=True, early_slack=2, per_frame=True)
        assert np.array_equal(o.cpu().numpy().reshape(4 * w, c.n), ref["hard"])
        assert np.array_equal(it.cpu().numpy(), np.asarray(ref["iters"]).reshape(-1))
    with pytest.raises(LdpcError):
        b.set_early_stop(False)
    b.close()


def test_resident_ctas_come_back(cuda):
    """As many CTAs as fit is what a batch asks for until it is given a number: that outlasts the toggling."""
    b = Batch(codes(), "OMS")
    auto = b.info()["ctas_per_sm"]
    b.set_early_stop(True)
    b.set_early_stop(False)
    assert b.info()["ctas_per_sm"] == auto
    b.configure(threads=128, ctas_per_sm=1)
    b.set_early_stop(True)
    assert b.info()["ctas_per_sm"] == 1
    b.close()
