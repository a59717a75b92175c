"""csrc/level_schedule.h on the CPU: for codes of several degrees, numbers of words and CTA rules, every
edge of every row is in one record, rows that share a variable keep their order with a barrier between
them, and no step reaches past its CTA, its messages or the limits of its records."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>
#include "level_schedule.h"
using namespace ldpc;
#define CHECK(x) if (!(x)) { printf("line %d: %s (n %d m %d words %lld)\n", __LINE__, #x, n, m, words); exit(1); }
static void check(int n, int m, const std::vector<int>& degrees, long long words, int fixed, bool may_half)
{
    std::mt19937 rng(n + m);
    std::vector<int32_t> ptr(1, 0), cols;
    std::vector<uint8_t> cls;
    for (int r = 0; r < m; r++) {
        std::set<int> v;
        while ((int)v.size() < degrees[r % degrees.size()]) v.insert(rng() % n);
        cols.insert(cols.end(), v.begin(), v.end());
        ptr.push_back((int)cols.size());
        cls.push_back(r >= m / 2);
    }
    const Rows H{n, m, ptr.data(), cols.data(), cls.data()};
    LevelSchedule s;
    const size_t lds = 4 * (size_t)n;
    if (!level_choose(H, lds, words, 148, fixed, may_half, s)) {
        CHECK(n > LEVEL_MAX_VARS);
        return;
    }
    const int per = s.fp == 1 && !s.half ? 2 : 1;
    CHECK(s.threads % 32 == 0 && s.threads <= 512 && (!fixed || s.threads == fixed));
    CHECK(may_half || !s.half);
    std::vector<int> row_of(cols.size()), seen(cols.size(), 0), last(n, -1), when(n, -1);
    for (int r = 0; r < m; r++)
        for (int e = ptr[r]; e < ptr[r + 1]; e++) row_of[e] = r;
    long long moff = 0;
    int barrier = 0;
    for (const LevelStep& t : s.steps) {
        const int nv = t.info & 0xff, lgs = (t.info >> 8) & 0xff, first = t.info >> 20;
        CHECK(nv >= 1 && nv <= 8 && lgs <= 2 && t.cnt % (1 << lgs) == 0);
        CHECK(t.cnt * per <= s.threads && first % 32 == 0 && first < s.threads);
        CHECK(t.moff == moff && t.moff % 16 == 0);
        moff += (4ll * nv * t.cnt + 15) / 16 * 16;
        CHECK(t.rec0 + t.cnt <= (int)s.recs.size());
        for (int k = t.rec0; k < t.rec0 + t.cnt; k++) {
            const uint4 q = s.recs[k];
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
            const int d = nv - (int)((q.x >> 1) & 1);
            CHECK(d >= 1);
            const int row = row_of[s.edges[8 * k]];
            for (int j = 0; j < 8; j++) {
                const int e = s.edges[8 * k + j];
                CHECK((e >= 0) == (j < d));
                if (e < 0) continue;
                uint32_t off = (w[j >> 1] >> (16 * (j & 1))) & 0xffffu;
                if (j == 0) off &= 0xfffcu;
                CHECK(off == 4u * cols[e] && row_of[e] == row && (q.x & 1) == cls[row] && !seen[e]++);
                CHECK(row_of[s.edges[8 * (t.rec0 + ((k - t.rec0) >> lgs << lgs))]] == row);
                const int v = cols[e];
                CHECK(last[v] < row && when[v] < barrier);  // in table order, a barrier in between
                last[v] = row;
                when[v] = barrier;
            }
        }
        barrier += (t.info >> 16) & 1;
    }
    CHECK(moff == s.msg_bytes);
    for (int x : seen) CHECK(x == 1);
}
int main()
{
    for (long long words : {1ll, 2ll, 74ll, 148ll, 149ll, 20000ll})
        for (int fixed : {0, 128, 256})
            for (int half = 0; half < (fixed ? 1 : 2); half++) {
                check(576, 288, {6}, words, fixed, half);
                check(4000, 2000, {6}, words, fixed, half);
                check(2304, 1152, {7, 6}, words, fixed, half);
                check(1944, 5, {7}, words, fixed, half);
                check(301, 120, {1, 2, 3, 4, 5, 8, 9, 13, 16, 17, 19}, words, fixed, half);
                check(2048, 384, {32}, words, fixed, half);
                check(816, 408, {10}, words, fixed, half);
                check(16384, 900, {3, 31}, words, fixed, half);
                check(16385, 300, {6}, words, fixed, half);
            }
    return 0;
}
"""


def test_schedules_hold(tmp_path):
    src = tmp_path / "t.cu"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.check_call([os.environ.get("NVCC", "nvcc"), "-O1", "-std=c++17", "-w", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", os.path.join(ROOT, "fast_ldpc_decoder_for_gpu_fixed_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"), "-o", exe, str(src)])
    run = subprocess.run([exe], timeout=120, capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
