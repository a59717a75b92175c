"""csrc/host_pipe.h: the helper threads of a host decode while the caller waits for the GPU.  They take no
core for the length of the wait, and the next shared loop finds them all, however long they had nothing to
do.  Runs without a GPU."""
import os
import subprocess

import pytest

from test_host_pipe_fork import CUDA, ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <sys/resource.h>
#include <unistd.h>
#include "host_pipe.h"
static double cpu_ms()
{
    rusage u;
    getrusage(RUSAGE_SELF, &u);
    return 1e3 * (u.ru_utime.tv_sec + u.ru_stime.tv_sec) + 1e-3 * (u.ru_utime.tv_usec + u.ru_stime.tv_usec);
}
int main(int argc, char** argv)
{
    ldpc::HostTeam team(atoi(argv[1]));
    // a long wait in the middle of a call
    team.wake();
    team.each([](int, int) {});
    const double before = cpu_ms();
    usleep(400000);
    const double idle = cpu_ms() - before;
    team.rest();
    team.wake();
    if (idle > 100.0) {
        printf("%.0f ms of CPU time in a wait of 400 ms\n", idle);
        team.rest();
        return 2;
    }
    // loops after waits of all lengths, over several calls; every part runs once a loop
    long sums[16] = {0}, loops = 0;
    unsigned r = 1;
    for (int call = 0; call < 20; call++) {
        if (call) team.wake();
        for (int i = 0; i < 60; i++, loops++) {
            r = r * 1664525u + 1013904223u;
            if (r >> 31) usleep((r >> 8) % 400);
            team.each([&](int part, int parts) { sums[part] += parts; });
        }
        team.rest();
        if (call % 3 == 0) usleep(500);
    }
    for (int i = 0; i < team.size(); i++)
        if (sums[i] != loops * team.size()) return 3;
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pipe")
    src, exe = d / "t.cpp", str(d / "t")
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", str(src), "-o", exe,
                           "-I", os.path.join(ROOT, "fast_ldpc_decoder_for_gpu_fixed_b200", "csrc"),
                           "-I", os.path.join(CUDA, "include"), "-L", os.path.join(CUDA, "lib64"),
                           "-lcudart_static", "-ldl", "-lrt"])
    return exe


@pytest.mark.parametrize("helpers", [0, 1, 3, 5])
def test_helpers_rest_during_a_wait(program, helpers):
    run = subprocess.run([program, str(helpers)], timeout=60, capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
