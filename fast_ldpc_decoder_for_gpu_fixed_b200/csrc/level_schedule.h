// Host side of decode_level_bytes_kernel (level_kernel.cuh): the order of a code's rows as steps
// that share no variable, the records of their lanes, and the choice of the CTA's shape.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

#include "level_kernel.cuh"

namespace ldpc {

// H as CSR rows in the reference's serial order
struct Rows {
    int n, m;
    const int32_t* ptr;
    const int32_t* cols;
    const uint8_t* cls;
    int degree(int r) const { return ptr[r + 1] - ptr[r]; }
};

struct LevelSchedule {
    std::vector<uint4> recs;
    std::vector<LevelStep> steps;
    std::vector<int32_t> edges;  // [8 * record + j]
    int msg_bytes = 0;
    int fp = 2, threads = 0;  // frame pairs per thread, CTA width
    bool half = false;        // one frame pair per CTA (fp = 1)
};

// lanes of a row (as a shift): at most 8 edges a lane
inline int level_lane_bits(int degree) { return degree <= 8 ? 0 : (degree <= 16 ? 1 : 2); }

// Rows in the order of their steps: step i is rows[end[i - 1]] .. rows[end[i] - 1].
struct LevelSteps {
    std::vector<int> rows, end;
    void swap(LevelSteps& o) { rows.swap(o.rows), end.swap(o.end); }
};

// Which rows wait for which: only rows that share a variable must keep their order.
class LevelOrder {
public:
    explicit LevelOrder(const Rows& H) : H_(H), preds_(H.m, 0), height_(H.m, 1), head_(H.m, -1)
    {
        std::vector<int> last(H.n, -1);
        link_.reserve(H.ptr[H.m]);
        for (int r = 0; r < H.m; r++) {
            same_degree_ = same_degree_ && H.degree(r) == H.degree(0);
            for (int e = H.ptr[r]; e < H.ptr[r + 1]; e++) {
                int& l = last[H.cols[e]];
                if (l == r) repeated = true;
                if (l >= 0 && l != r) {
                    link_.push_back({r, head_[l]});
                    head_[l] = (int)link_.size() - 1;
                    preds_[r]++;
                }
                l = r;
            }
        }
        for (int r = H.m - 1; r >= 0; r--) {
            for (int k = head_[r]; k >= 0; k = link_[k].next) height_[r] = std::max(height_[r], height_[link_[k].row] + 1);
            top_ = std::max(top_, height_[r]);
        }
    }
    bool repeated = false;  // a row holds a variable twice: its edges have an order
    int least() const { return top_; }  // the fewest steps

    // Steps of at most `most` lanes, the rows with the longest chain of followers first.  A row
    // may wait for a later step than the first it could take (ldpc_code::levels): that fills the
    // warps (4000x2000 with 96 lanes: 67 warps an iteration instead of 75 in the same 26 steps,
    // and 3 instead of 5 of them at once).
    void steps(int most, LevelSteps& out) const
    {
        std::vector<int> preds(preds_), bucket(top_ + 1, -1), below(H_.m);  // ready rows by height
        auto push = [&](int r) {
            below[r] = bucket[height_[r]];
            bucket[height_[r]] = r;
        };
        for (int r = H_.m - 1; r >= 0; r--)
            if (!preds[r]) push(r);
        out.rows.clear();
        out.end.clear();
        out.rows.reserve(H_.m);
        int top = top_;
        while ((int)out.rows.size() < H_.m) {
            const int first = (int)out.rows.size();
            int used = 0, h = top;
            for (; h > 0; h--)
                while (bucket[h] >= 0) {
                    const int r = bucket[h], lanes = 1 << level_lane_bits(H_.degree(r));
                    if (used && used + lanes > most) goto full;
                    used += lanes;
                    bucket[h] = below[r];
                    out.rows.push_back(r);
                }
        full:
            while (top > 0 && bucket[top] < 0) top--;
            for (int i = first; i < (int)out.rows.size(); i++)
                for (int k = head_[out.rows[i]]; k >= 0; k = link_[k].next)
                    if (--preds[link_[k].row] == 0) {
                        push(link_[k].row);
                        top = std::max(top, height_[link_[k].row]);
                    }
            if (!same_degree_)
                std::stable_sort(out.rows.begin() + first, out.rows.end(), [&](int a, int b) { return H_.degree(a) > H_.degree(b); });
            out.end.push_back((int)out.rows.size());
        }
    }

private:
    struct Link {
        int row, next;
    };
    const Rows& H_;
    std::vector<int> preds_, height_, head_;
    std::vector<Link> link_;
    int top_ = 0;
    bool same_degree_ = true;
};

// Calls f(r0, r1, lgs, nv, last) for each part [r0, r1) of the steps whose rows share the lanes per
// row (1 << lgs) and, but for one, the edges per lane (nv); last: the part ends its step.
template <class F>
void level_parts(const Rows& H, const LevelSteps& S, F f)
{
    int r0 = 0;
    for (int end : S.end)
        while (r0 < end) {
            const int d = H.degree(S.rows[r0]), lgs = level_lane_bits(d), nv = (d + (1 << lgs) - 1) >> lgs;
            int r1 = r0;
            while (r1 < end && level_lane_bits(H.degree(S.rows[r1])) == lgs && H.degree(S.rows[r1]) >> lgs >= nv - 1) r1++;
            f(r0, r1, lgs, nv, r1 == end);
            r0 = r1;
        }
}

// The records of the steps.  The edges of a row are dealt to its lanes and positions so that the
// 32 APP words a warp touches together fall into different shared-memory banks as far as that
// goes: a row's edges have no order (its minima and parity do not depend on it).  With random
// columns in table order the 32 words take about 3.5 passes, dealt out like this 2.0.
inline void level_records(const Rows& H, const LevelSteps& order, LevelSchedule& out)
{
    const int per = out.fp == 1 && !out.half ? 2 : 1, group = 32 / per;  // threads of a record, records of a warp
    const std::vector<int>& rows = order.rows;
    long long moff = 0;
    level_parts(H, order, [&](int r0, int r1, int lgs, int nv, bool last) {
        const int S = 1 << lgs, rec0 = (int)out.recs.size(), lanes = (r1 - r0) << lgs;
        out.steps.push_back({rec0, (int)moff, lanes, nv | lgs << 8 | (int)last << 16});
        moff += (4ll * nv * lanes + 15) / 16 * 16;
        out.recs.resize(rec0 + lanes, make_uint4(0, 0, 0, 0));
        out.edges.resize(8 * out.recs.size(), -1);
        for (int w0 = r0; w0 < r1; w0 += group >> lgs) {
            const int w1 = std::min(r1, w0 + (group >> lgs));
            uint8_t cnt[8][32] = {};  // [position][bank] of this warp
            int at[32][32];           // [row][lane * nv + position]: its edge or -1
            for (int i = w0; i < w1; i++) {
                const int d = H.degree(rows[i]);
                for (int p = 0; p < S * nv; p++) {
                    const int e = p / nv + (p % nv) * S;  // lane s holds edges s, s + S, ...
                    at[i - w0][p] = e < d ? e : -1;
                    if (e < d) cnt[p % nv][H.cols[H.ptr[rows[i]] + e] & 31]++;
                }
            }
            for (int i = w0; i < w1; i++) {
                const int32_t* cols = H.cols + H.ptr[rows[i]];
                int* a = at[i - w0];
                for (int p = 0; p < S * nv; p++)
                    for (int q = p + 1; q < S * nv; q++) {
                        if (a[p] < 0 || a[q] < 0) continue;
                        uint8_t *cp = cnt[p % nv], *cq = cnt[q % nv];
                        const int bp = cols[a[p]] & 31, bq = cols[a[q]] & 31;
                        // swap the two where that leaves fewer collisions
                        if (cp == cq || bp == bq || cp[bq] + cq[bp] + 2 >= cp[bp] + cq[bq]) continue;
                        cp[bp]--, cq[bq]--, cp[bq]++, cq[bp]++;
                        std::swap(a[p], a[q]);
                    }
            }
            for (int i = w0; i < w1; i++)
                for (int s = 0; s < S; s++) {
                    const int* a = &at[i - w0][s * nv];
                    const size_t k = (size_t)rec0 + ((size_t)(i - r0) << lgs) + s;
                    uint32_t w[4] = {0, 0, 0, 0};
                    for (int j = 0; j < nv; j++) {
                        if (a[j] < 0) {
                            w[0] |= 2u;  // nv - 1 edges
                            continue;
                        }
                        const int e = H.ptr[rows[i]] + a[j];
                        w[j >> 1] |= (uint32_t)(4 * H.cols[e]) << (16 * (j & 1));
                        out.edges[8 * k + j] = e;
                    }
                    if (H.cls[rows[i]]) w[0] |= 1u;
                    out.recs[k] = make_uint4(w[0], w[1], w[2], w[3]);
                }
        }
    });
    // each step starts on the warp after the last one of the step before, so that narrow steps
    // do not leave the same warps (and their quarter of the SM) idle every time
    int at = 0;
    for (auto& st : out.steps) {
        st.info |= at << 20;
        at = (at + (st.cnt * per + 31) / 32 * 32) % out.threads;
    }
    out.msg_bytes = (int)std::min(moff, 1ll << 30);
}

// Chooses steps, frame pairs per thread and CTA width for `words` words on `sms` multiprocessors,
// by the cycles an iteration of one word takes its SM: the issue slots of its warps (about 300
// instructions a full warp of rows with two pairs a thread, 185 with one, 30 an idle one, over
// four schedulers, which a width that is not a multiple of 128 loads unevenly) plus the latency
// of its steps (580 cycles up to 128 threads, 60 more for each further 128; 100 less with one
// pair a thread) shared by the words that are resident together.  Measured (us): 4000x2000, 1024
// words: two pairs, steps of 96 lanes and 128 threads 624, 96 threads 653, 128 lanes 645, 64
// lanes 627, one pair 674; 1944x972, 777 words: 96 threads (6 words a multiprocessor, one round)
// 478, 128 threads (5) 520; 576x288, one word: one pair 68, two pairs 88; 2304x1152, 1024 words:
// 96 lanes 229, 192 lanes 236, one word: 42 and 40.  The registers a thread (72, 96) are those of the
// two-pair kernels without the early stop; with it they take up to 122 (per frame), so there the rule
// counts more words as resident than are, and its cost is the lower bound of it.
// Host time to choose and lay out a schedule: 0.1 ms for 576x288, 0.7 for 4000x2000, 2.2 for 9972x4986.
// lds: shared memory beside the messages; fixed_threads: the CTA width, 0 = free; may_half: one
// frame pair per CTA is allowed (it pays while the words leave multiprocessors idle).  False when
// the code has no such schedule.
inline bool level_choose(const Rows& H, size_t lds, long long words, int sms, int fixed_threads, bool may_half,
                         LevelSchedule& out)
{
    if (H.n > LEVEL_MAX_VARS) return false;
    LevelOrder order(H);
    if (order.repeated) return false;
    LevelSteps best, cur;
    bool uniform = true;
    for (int r = 1; r < H.m && uniform; r++) uniform = H.degree(r) == H.degree(0);
    const int regs = uniform && (H.degree(0) == 6 || H.degree(0) == 7) ? 72 : 96;
    double best_cost = 0;
    size_t last_steps = 0;
    const int widths[] = {32, 64, 96, 128, 256};
    // the widest that the CTA allows is always considered, so that a wide code has a schedule at any
    // width of the batch's persistent kernel (short irregular codes and a Z = 256 code, 12 500 words,
    // early stop, 128 threads: 1.86 ms; 7.70 ms on the per-byte kernel that serves a batch without one)
    int widest_most = 256;
    for (int most : widths)
        if (!fixed_threads || most <= fixed_threads) widest_most = most;
    for (int most : widths) {
        if (most > widest_most) break;
        // too narrow for the code: many more steps than its longest chain
        if (most < widest_most && (long long)most * order.least() * 3 < 2ll * H.m) continue;
        order.steps(most, cur);
        if (last_steps == cur.end.size()) break;  // no step is wider than before
        last_steps = cur.end.size();
        bool used = false;
        for (int mode = 0; mode < (fixed_threads ? 1 : (may_half ? 3 : 2)); mode++) {
            const int fp = mode == 0 ? 2 : 1, per = mode == 1 ? 2 : 1;
            long long warps = 0, steps = 0, bytes = 0;
            int widest = 0;
            level_parts(H, cur, [&](int r0, int r1, int lgs, int nv, bool) {
                const int lanes = (r1 - r0) << lgs;
                steps++;
                warps += (lanes * per + 31) / 32;
                bytes += (4ll * nv * lanes + 15) / 16 * 16;
                widest = std::max(widest, lanes * per);
            });
            if (widest > 512) continue;
            for (int T : {(widest + 31) / 32 * 32, (widest + 127) / 128 * 128}) {
                if (fixed_threads) T = fixed_threads;
                const long long idle = steps * (T / 32) - warps, ctas = mode == 2 ? 2 * words : words;
                const long long fit = std::max<long long>(
                    1, std::min<long long>(227 * 1024 / (long long)(lds + bytes + 1024), 65536 / (T * regs)));
                const long long per_sm = (ctas + sms - 1) / sms, rounds = (per_sm + fit - 1) / fit;
                const double issue = (warps * (fp == 2 ? 300.0 : 185.0) + idle * 30.0) / 4 * (T > 64 && T % 128 ? 1.1 : 1.0);
                const double latency = steps * ((fp == 2 ? 520.0 : 420.0) + 60.0 * ((T + 127) / 128));
                const double cost = issue * per_sm + latency * rounds;
                if (best_cost == 0 || cost < best_cost) {
                    best_cost = cost;
                    out.fp = fp;
                    out.half = mode == 2;
                    out.threads = T;
                    used = true;
                }
            }
        }
        if (used) best.swap(cur);
    }
    if (best_cost == 0) return false;
    level_records(H, best, out);
    return out.steps.size() <= (size_t)LEVEL_MAX_STEPS && out.msg_bytes < (1 << 20);
}

}  // namespace ldpc
