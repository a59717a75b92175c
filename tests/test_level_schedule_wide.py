"""csrc/level_schedule.h on the CPU for wide, shallow codes (a few levels of hundreds of rows) at a given
CTA width, as the batch's persistent kernel asks for it: there is a schedule of that width, and it holds
what test_level_schedule.py asks of every schedule."""
import os
import subprocess

import pytest

from test_level_schedule import PROGRAM, ROOT

MAIN = r"""
int main(int argc, char** argv)
{
    const int fixed = atoi(argv[1]);
    for (long long words : {1ll, 1ll << 30}) {
        check(16384, 4000, {2}, words, fixed, false);
        check(16384, 3000, {3}, words, fixed, false);
        check(16384, 1500, {2, 3, 5}, words, fixed, false);
        check(16384, 1200, {9, 17, 2}, words, fixed, false);
        check(4096, 600, {2, 4}, words, fixed, false);
        check(1024, 256, {1, 2}, words, fixed, false);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("wide")
    src, exe = d / "t.cu", str(d / "t")
    src.write_text(PROGRAM.split("int main()")[0] + MAIN)
    subprocess.check_call([os.environ.get("NVCC", "nvcc"), "-O1", "-std=c++17", "-w", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", os.path.join(ROOT, "fast_ldpc_decoder_for_gpu_fixed_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"), "-o", exe, str(src)])
    return exe


@pytest.mark.parametrize("fixed", range(32, 257, 32))
def test_wide_codes_have_a_schedule(program, fixed):
    run = subprocess.run([program, str(fixed)], timeout=120, capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
