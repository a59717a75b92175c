"""csrc/host_pipe.h in a forked child: the child frees its copy of a decoder while a pipe is idle.

The pipe's threads exist in the parent only, so a child that took the pipe apart would wait for them
for good.  Runs without a GPU: the pipe is made without its pinned memory and events.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include <sys/wait.h>
#include <unistd.h>
#include "host_pipe.h"
int main(int argc, char** argv)
{
    using namespace ldpc;
    HostPipes::user(1);
    HostPipe* p = new HostPipe(%d, 0);
    long sums[8] = {0};
    p->team.wake();
    for (int r = 0; r < 50; r++) p->team.each([&](int part, int parts) { sums[part] += parts; });
    p->team.rest();
    for (int i = 0; i < p->team.size(); i++)
        if (sums[i] != 50L * p->team.size()) return 3;
    HostPipes::give(p);
    const pid_t child = fork();
    if (child == 0) {
        HostPipes::user(-1);
        _exit(0);
    }
    for (int i = 0; i < 200; i++) {
        int st = 0;
        if (waitpid(child, &st, WNOHANG) == child) {
            HostPipes::user(-1);  // the parent's pipe goes here
            return WIFEXITED(st) && WEXITSTATUS(st) == 0 ? 0 : 4;
        }
        usleep(50000);
    }
    kill(child, SIGKILL);
    waitpid(child, nullptr, 0);
    return 5;
}
"""


@pytest.mark.parametrize("helpers", [0, 1, 3])
def test_fork_with_an_idle_pipe(tmp_path, helpers):
    src = tmp_path / "t.cpp"
    src.write_text("#include <csignal>\n" + PROGRAM % helpers)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", str(src), "-o", exe,
                           "-I", os.path.join(ROOT, "fast_ldpc_decoder_for_gpu_fixed_b200", "csrc"),
                           "-I", os.path.join(CUDA, "include"), "-L", os.path.join(CUDA, "lib64"),
                           "-lcudart_static", "-ldl", "-lrt"])
    assert subprocess.run([exe], timeout=60).returncode == 0
