// Level-scheduled decoder with byte storage and fp16x2 arithmetic.
//
// State (shared memory, 4 frames = one reference word per CTA): the APP as one byte per
// variable and frame, b = 127 - x (word v holds the 4 frames of variable v), and the
// messages as one byte per edge and frame, mu = 128 + m with m the negated message.  A
// thread turns the bytes of an edge into fp16x2 lanes with one byte permute per frame pair
// (the byte under 0x64 is the fp16 1024 + byte) and does the row arithmetic of namespace h2
// on them, so a row costs half the shared-memory traffic of fp16 storage and a third of the
// instructions of per-byte SIMD intrinsics, which the hardware emulates.
//
// What bounds it: a full warp of degree-6 rows issues about 300 instructions, 130 of them on
// the ALU pipe (half rate: HMNMX2, PRMT, LOP3) and 105 on the fp16 pipe (half rate), so
// 4000x2000 needs 53 us per word and 20 iterations of its multiprocessor; the rest of the 83 us
// it takes (4440 words) is latency that 3 resident words of 4 warps do not cover.  Measured, OMS,
// 20 iterations, us before (fp16 storage, 2 frames per CTA, table-order levels) and now:
// 4000x2000, 1024 words 1001 / 628; 1944x972 NMS, 30 iterations, 777 words 797 / 479; 2304x1152
// 2NMS (byte SIMD before), 1500 words 641 / 281; 9972x4986 early stop (byte SIMD before), 501
// words 932 / 511; 576x288, one word 127 / 68.  With half the message area (wrong results, timing
// only) and 6 words resident, 4000x2000 takes 70 us a word: shared memory is what limits it.
#pragma once
#include "decode_kernel.cuh"

namespace ldpc {

// One step of the schedule: rows of one level that share the number of lanes per row
// (1 << lgs) and the number of edges per lane (nv; a lane may hold nv - 1).  Packed so that a
// step is one uniform 16-byte load.
struct LevelStep {
    int rec0;  // first record
    int moff;  // byte offset of the step's messages behind the APP
    int cnt;   // records (rows << lgs), at most one per thread (two threads each with FP = 1)
    int info;  // nv | lgs << 8 | (the level ends here: a barrier) << 16 | first thread << 20
};

// Record of one lane of a row: byte offsets 4 * v of its edges' APP words.  Bit 0 of the
// first: the row's class; bit 1: the lane holds nv - 1 edges.
struct LevelPlan {
    const uint4* rec;
    const LevelStep* step;
    const int32_t* edge;  // [8 * record + j]: the edge's index in table order (state dumps)
    int nstep;
    int msg_bytes;  // all messages of the 4 frames
    uint32_t c64 = 0x64646464u, c128 = 0x58005800u;  // lv::Regs
};

constexpr int LEVEL_MAX_VARS = 16384;  // 4 * v fits 16 bits
constexpr int LEVEL_MAX_STEPS = 1024;  // odd-row counts per lane stay exact in fp16

namespace lv {

// Constants that instructions need in a register beside an immediate.  They come from the kernel's
// parameters because the compiler moves known constants into place before each use (one move for
// every other byte permute).
struct Regs {
    uint32_t c64, c128;
    __device__ __forceinline__ Regs(uint32_t a, uint32_t b) : c64(a), c128(b) {}
};
constexpr uint32_t C1152 = 0x64806480u;

__device__ __forceinline__ uint32_t off(const uint4& r, int j)
{
    const uint32_t w = j < 2 ? r.x : (j < 4 ? r.y : (j < 6 ? r.z : r.w));
    return j == 0 ? (w & 0xfffcu) : ((j & 1) ? w >> 16 : (w & 0xffffu));
}

// NV elements of FP * 2 bytes of lane i: 16-, 8-, 4- and 2-byte parts, each an array over the
// step's lanes, so that every access of a warp is contiguous.
template <int NV, int FP>
struct Msg {
    static constexpr int BYTES = NV * FP * 2;
    static constexpr int W = (BYTES + 3) / 4;
    // byte offset of the part that starts at byte b of an element list, lane i
    __device__ __forceinline__ static void load(const char* p, int lanes, int i, uint32_t (&m)[W])
    {
        int b = 0, w = 0;
#pragma unroll
        for (; b + 16 <= BYTES; b += 16, w += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(p + b * lanes + 16 * i);
            m[w] = v.x, m[w + 1] = v.y, m[w + 2] = v.z, m[w + 3] = v.w;
        }
        if (BYTES & 8) {
            const uint2 v = *reinterpret_cast<const uint2*>(p + b * lanes + 8 * i);
            m[w] = v.x, m[w + 1] = v.y;
            b += 8, w += 2;
        }
        if (BYTES & 4) {
            m[w] = *reinterpret_cast<const uint32_t*>(p + b * lanes + 4 * i);
            b += 4, w += 1;
        }
        if (BYTES & 2) m[w] = *reinterpret_cast<const uint16_t*>(p + b * lanes + 2 * i);
    }
    __device__ __forceinline__ static void store(char* p, int lanes, int i, const uint32_t (&m)[W])
    {
        int b = 0, w = 0;
#pragma unroll
        for (; b + 16 <= BYTES; b += 16, w += 4)
            *reinterpret_cast<uint4*>(p + b * lanes + 16 * i) = make_uint4(m[w], m[w + 1], m[w + 2], m[w + 3]);
        if (BYTES & 8) {
            *reinterpret_cast<uint2*>(p + b * lanes + 8 * i) = make_uint2(m[w], m[w + 1]);
            b += 8, w += 2;
        }
        if (BYTES & 4) {
            *reinterpret_cast<uint32_t*>(p + b * lanes + 4 * i) = m[w];
            b += 4, w += 1;
        }
        if (BYTES & 2) *reinterpret_cast<uint16_t*>(p + b * lanes + 2 * i) = (uint16_t)m[w];
    }
};

// KIND_LEARNED magnitude tables: 128 fp16 values per row class
__device__ __forceinline__ uint32_t lut2(uint32_t a, const uint16_t* lut)
{
    const uint32_t r = h2::add(a, h2::C1024);
    return (uint32_t)lut[r & 0xffu] | ((uint32_t)lut[(r >> 16) & 0xffu] << 16);
}

// The update of one row (or, with SPLIT, of a lane's part of it) for FP frame pairs.  B[p][j] =
// 1024 + b and M[p][j] = 1152 + m in, the new ones out; odd[p]: the sign bits set in the lanes
// whose row is odd.  MIXED: only the first d edges are there.  The pairs are written side by side: their chains are independent, and one
// warp alone would wait on most of its instructions.
template <int KIND, int NV, int FP, int PER, bool SPLIT, bool MIXED = false>
__device__ __forceinline__ void row_pairs(const Regs& R, uint32_t (&B)[FP][NV], uint32_t (&M)[FP][NV], bool shortrow,
                                          int lgs, unsigned wmask, bool noclip, const uint16_t* lut, uint32_t (&odd)[FP],
                                          int d = NV)
{
    using namespace h2;
    uint32_t ut[FP][NV], mn1[FP], mn2[FP];
#pragma unroll
    for (int j = 0; j < NV; j++)
#pragma unroll
        for (int p = 0; p < FP; p++) {
            // clamp(b - m, 0, 255) from 1024 + b and 1152 + m (their difference is exact)
            B[p][j] = hmin(fma_relu(sub(B[p][j], M[p][j]), ONE, R.c128), C255);
            ut[p][j] = add(B[p][j], CNEG127);
        }
#pragma unroll
    for (int p = 0; p < FP; p++) {
        // no such edge: the neutral magnitude and sign
        if (SPLIT && shortrow) ut[p][NV - 1] = C127;
#pragma unroll
        for (int j = 0; j < NV; j++)
            if (MIXED && j >= d) ut[p][j] = C127;
        mn1[p] = NV == 1 ? ut[p][0] : min_xs(ut[p][0], ut[p][NV > 1 ? 1 : 0]);
        mn2[p] = NV == 1 ? C127 : max_xs(ut[p][0], ut[p][NV > 1 ? 1 : 0]);
    }
#pragma unroll
    for (int j = 2; j + 1 < NV; j += 2)
#pragma unroll
        for (int p = 0; p < FP; p++) {
            const uint32_t lo = min_xs(ut[p][j], ut[p][j + 1]), hi = max_xs(ut[p][j], ut[p][j + 1]);
            const uint32_t x = max_xs(mn1[p], lo), y = min_xs(mn2[p], hi);
            // the last one by magnitude alone: the sign of min2 is not used, and the abs is free here
            mn2[p] = j + 2 >= NV ? hmin(habs(x), habs(y)) : min_xs(x, y);
            mn1[p] = min_xs(mn1[p], lo);
        }
#pragma unroll
    for (int p = 0; p < FP; p++) {
        if ((NV & 1) && NV > 1) {
            const uint32_t mx = max_xs(ut[p][NV - 1], mn1[p]);
            mn1[p] = min_xs(mn1[p], ut[p][NV - 1]);
            mn2[p] = hmin(habs(mn2[p]), habs(mx));
        }
    }
    if (SPLIT)
        for (int o = PER; o < (PER << lgs); o <<= 1)
#pragma unroll
            for (int p = 0; p < FP; p++) {
                const uint32_t p1 = __shfl_xor_sync(wmask, mn1[p], o), p2 = __shfl_xor_sync(wmask, mn2[p], o);
                mn2[p] = hmin(hmin(habs(mn2[p]), habs(p2)), habs(max_xs(mn1[p], p1)));
                mn1[p] = min_xs(mn1[p], p1);
            }
    uint32_t c1s[FP], dcs[FP];
#pragma unroll
    for (int p = 0; p < FP; p++) {
        // the minima start at 127 in the reference; |t| reaches 128 only for x = -128, which shows
        // only where magnitudes are not clipped to 31
        if (KIND == KIND_NMS || KIND == KIND_2NMS || KIND == KIND_LEARNED || (KIND == KIND_OMS && noclip)) {
            mn1[p] = min_xs(mn1[p], C127);
            mn2[p] = min_xs(mn2[p], C127);
        }
        odd[p] = mn1[p] & SIGN;
        const uint32_t a2 = NV >= 3 ? mn2[p] : habs(mn2[p]);
        uint32_t c1, c2;
        if (KIND == KIND_LEARNED) {
            c1 = lut2(a2, lut);
            c2 = lut2(habs(mn1[p]), lut);
        } else {
            mags<KIND>(habs(mn1[p]), a2, noclip, c1, c2, 0, 0);
        }
        c1s[p] = c1 | odd[p];
        dcs[p] = sub(c2 | odd[p], c1s[p]);
    }
#pragma unroll
    for (int j = 0; j < NV; j++)
#pragma unroll
        for (int p = 0; p < FP; p++) {
            const uint32_t r = fma(sub_sat(habs(ut[p][j]), habs(mn1[p])), dcs[p], c1s[p]);
            const uint32_t mo = r ^ (ut[p][j] & SIGN);
            M[p][j] = add(mo, C1152);
            B[p][j] = add(hmin(fma_relu(mo, ONE, B[p][j]), C255), C1024);
        }
}

// Updates lane i of a step.  FP = 2: the thread does the 4 frames of the word; FP = 1: the pair at
// byte h of the words (PER = 2: lanes 2k and 2k + 1 do frames 0, 1 and 2, 3 of record k).
template <int KIND, int NV, int FP, int PER, bool SPLIT>
__device__ __forceinline__ void row(const Regs& R, char* app, char* msg, int lanes, int i, int h, const uint4& rec, int lgs, unsigned wmask,
                                    bool noclip, const uint16_t* lut, uint32_t (&odd)[FP])
{
    const bool shortrow = SPLIT && (rec.x & 2u);
    uint32_t w[NV], mw[Msg<NV, FP>::W];
#pragma unroll
    for (int j = 0; j < NV; j++)
        w[j] = FP == 2 ? *reinterpret_cast<const uint32_t*>(app + off(rec, j))
                       : *reinterpret_cast<const uint16_t*>(app + off(rec, j) + h);
    Msg<NV, FP>::load(msg, lanes, i, mw);
    uint32_t B[FP][NV], M[FP][NV];
#pragma unroll
    for (int j = 0; j < NV; j++)
#pragma unroll
        for (int p = 0; p < FP; p++) {
            B[p][j] = __byte_perm(w[j], R.c64, p == 0 ? 0x4140 : 0x4342);
            M[p][j] = FP == 2 ? __byte_perm(mw[j], R.c64, p == 0 ? 0x4140 : 0x4342)
                              : __byte_perm(mw[j / 2], R.c64, (j & 1) ? 0x4342 : 0x4140);
        }
    row_pairs<KIND, NV, FP, PER, SPLIT>(R, B, M, shortrow, lgs, wmask, noclip, lut, odd);
#pragma unroll
    for (int j = 0; j < NV; j++) {
        if (FP == 2) {
            mw[j] = __byte_perm(M[0][j], M[FP - 1][j], 0x6420);
            if (!(SPLIT && j == NV - 1 && shortrow))
                *reinterpret_cast<uint32_t*>(app + off(rec, j)) = __byte_perm(B[0][j], B[FP - 1][j], 0x6420);
        } else {
            if (j & 1) mw[j / 2] = __byte_perm(M[0][j - (j & 1)], M[0][j], 0x6420);
            if (j == NV - 1 && !(j & 1)) mw[j / 2] = __byte_perm(M[0][j], 0, 0x4420);
            if (!(SPLIT && j == NV - 1 && shortrow))
                *reinterpret_cast<uint16_t*>(app + off(rec, j) + h) = (uint16_t)__byte_perm(B[0][j], 0, 0x4420);
        }
    }
    Msg<NV, FP>::store(msg, lanes, i, mw);
}

// bit 7 of each byte: that frame's hard decision (x > 0, that is b < 127) is 0
__device__ __forceinline__ uint32_t zero_bits(uint32_t b) { return b | ((b & 0x7f7f7f7fu) + 0x01010101u); }

// bit 7 of byte k is set in some thread when frame k has a check of odd parity
__device__ __forceinline__ uint32_t odd_checks(const LevelPlan& L, const char* app)
{
    uint32_t bad = 0;
    for (int s = 0; s < L.nstep; s++) {
        const int4 st = __ldg(reinterpret_cast<const int4*>(L.step) + s);
        const int nv = st.w & 0xff, lgs = (st.w >> 8) & 0xff;
        for (int k = threadIdx.x; k < st.z; k += blockDim.x) {
            const uint4 rec = __ldg(L.rec + st.x + k);
            const int d = nv - ((rec.x >> 1) & 1);
            // x > 0 edges: d minus the zero bits, so the parity of the zero bits and of d
            uint32_t acc = (d & 1) ? 0x80808080u : 0u;
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (j < d) acc ^= zero_bits(*reinterpret_cast<const uint32_t*>(app + off(rec, j)));
            if (lgs) {
                const int left = st.z - (k & ~31);
                const unsigned m = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
                for (int o = 1; o < (1 << lgs); o <<= 1) acc ^= __shfl_xor_sync(m, acc, o);
            }
            bad |= acc;
        }
    }
    return bad & 0x80808080u;
}

__device__ __forceinline__ uint32_t ones(uint32_t b) { return (~zero_bits(b) >> 7) & 0x01010101u; }

// hard decisions of the frames of kmask (see write_group), from the byte APP
__device__ __forceinline__ void write_hard(const Plan& P, const Job& J, long long g, const char* app, int kmask)
{
    const int n = P.n;
    const long long lg = g - J.word0;
    const uint32_t* a = reinterpret_cast<const uint32_t*>(app);
    if (J.counts) count_group_errors(P, J, g, [&](int v) { return a[v] ^ 0x7f7f7f7fu; }, kmask);
    if (!J.out) return;
    if (J.out_packed || (n & 3)) {
        if (!J.out_packed) {
            uint8_t* o = reinterpret_cast<uint8_t*>(J.out) + 4 * lg * n;
            for (int v = threadIdx.x; v < n; v += blockDim.x) {
                const uint32_t h = ones(a[v]);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if ((kmask >> k) & 1) o[k * n + v] = (h >> (8 * k)) & 1;
            }
            return;
        }
        const int nb = (n + 7) >> 3;
        uint8_t* o = reinterpret_cast<uint8_t*>(J.out) + 4 * lg * nb;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) {
            uint32_t acc = 0;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                // the APP array is padded to 16 variables
                const uint4 v = *reinterpret_cast<const uint4*>(a + 8 * b + 4 * q);
                const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (8 * b + 4 * q + j < n) acc |= ones(x[j]) << (4 * q + j);
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                if ((kmask >> k) & 1) o[k * nb + b] = (acc >> (8 * k)) & 0xff;
        }
        return;
    }
    const int n4 = n >> 2;
    uint32_t* o32 = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(J.out) + 4 * lg * n);
    for (int q = threadIdx.x; q < n4; q += blockDim.x) {
        const uint4 v = *reinterpret_cast<const uint4*>(a + 4 * q);
        const uint32_t x[4] = {ones(v.x), ones(v.y), ones(v.z), ones(v.w)};
        uint32_t w[4];
        transpose4x4(x, w);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if ((kmask >> k) & 1) o32[k * n4 + q] = w[k];
    }
}

// the word's LLRs into the byte APP
__device__ __forceinline__ void read_word(const Plan& P, const Job& J, long long g, char* app)
{
    const int n = P.n;
    if (J.gen || J.interleaved || (n & 3)) {
        uint32_t* a = reinterpret_cast<uint32_t*>(app);
        read_group(P, J, g, [&](int v, uint32_t w) { a[v] = w ^ 0x7f7f7f7fu; });
        return;
    }
    const uint32_t* f0 = reinterpret_cast<const uint32_t*>(J.llr + (4 * (g - J.word0)) * (long long)n);
    const int n4 = n >> 2;
    constexpr int U = 4;  // loads of U trips in flight
    for (int q0 = threadIdx.x; q0 < n4; q0 += U * blockDim.x) {
        uint32_t a[U][4];
#pragma unroll
        for (int t = 0; t < U; t++) {
            const int q = q0 + t * blockDim.x;
            if (q < n4)
#pragma unroll
                for (int k = 0; k < 4; k++) a[t][k] = __ldg(f0 + k * n4 + q) ^ 0x7f7f7f7fu;
        }
#pragma unroll
        for (int t = 0; t < U; t++) {
            const int q = q0 + t * blockDim.x;
            if (q < n4) {
                uint32_t w[4];
                transpose4x4(a[t], w);
                *reinterpret_cast<uint4*>(app + 16 * q) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    }
}

}  // namespace lv

// Decodes word g, or with HALF its frames 2 half, 2 half + 1.  NVX: the edges of every row, 0 for
// any (steps of 1..8 edges a lane, rows over up to 4 lanes).  ET: 0 = fixed iterations (2NMS: its own rule), 1 = syndrome early
// stop per word, 2 = per frame.  Every thread of the CTA calls it; s_odd: four words.
template <int KIND, int NVX, int FP, int ET, bool HALF = false>
__device__ __forceinline__ void decode_word_bytes(const Plan& P, const LevelPlan& L, const Job& J, long long g, char* smem,
                                                  unsigned* s_odd, int half = 0)
{
    static_assert(!HALF || (FP == 1 && ET == 0 && KIND != KIND_2NMS), "one pair per CTA: fixed iterations");
    constexpr int PER = FP == 1 && !HALF ? 2 : 1;  // threads of a record
    using namespace lv;
    char* app = smem;
    char* msgs = smem + 4 * P.npad;
    uint16_t* slut = reinterpret_cast<uint16_t*>(msgs + L.msg_bytes);
    if (threadIdx.x < 4) s_odd[threadIdx.x] = 0;
    read_word(P, J, g, app);
    for (int i = threadIdx.x; i < L.msg_bytes / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(msgs)[i] = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);
    __syncthreads();

    const Regs R(L.c64, L.c128);
    int executed = 0;
    bool passed = false;
    unsigned live = 0xFu;
    int its[4] = {0, 0, 0, 0};
    const int4* steps = reinterpret_cast<const int4*>(L.step);
    // thread t takes lane i = t - (the step's first thread), modulo the CTA
    auto lane = [&](const int4& x) {
        const int i = (int)threadIdx.x - (x.w >> 20);
        return i < 0 ? i + (int)blockDim.x : i;
    };
    // the step descriptors two steps and the thread's record one step ahead of their use
    int4 st = __ldg(steps), nx = __ldg(steps + (L.nstep > 1 ? 1 : 0));
    int sp = L.nstep > 2 ? 2 : 0;
    uint4 rec = make_uint4(0, 0, 0, 0);
    int i = lane(st);
    if (i / PER < st.z) rec = __ldg(L.rec + st.x + i / PER);
    const int h = FP == 2 ? 0 : (HALF ? 2 * half : 2 * (threadIdx.x & 1));  // steps start on even threads
    for (int it = 0; it < J.iters; it++) {
        uint32_t odd_any = 0;           // 2NMS
        uint32_t cnt[FP];               // +1 per even row, -1 per odd row and lane
        int rows = 0;
#pragma unroll
        for (int p = 0; p < FP; p++) cnt[p] = 0;
        const bool quirk = J.quirk && it == 0;
        if (KIND == KIND_LEARNED) {
            const int t = it < J.lut_its ? it : J.lut_its - 1;
            for (int i = threadIdx.x; i < 256; i += blockDim.x)
                slut[i] = __half_as_ushort(__int2half_rn(J.lut[t * 256 + i]));
            __syncthreads();
        }
        for (int s = 0; s < L.nstep; s++) {
            uint4 nrec = make_uint4(0, 0, 0, 0);
            const int k = i / PER, ni = lane(nx), nk = ni / PER;
            if (nk < nx.z) nrec = __ldg(L.rec + nx.x + nk);
            const int4 nx2 = __ldg(steps + sp);
            sp = sp + 1 < L.nstep ? sp + 1 : 0;
            char* msg = msgs + st.y;
            if (k < st.z) {
                const int cls = rec.x & 1;
                const bool noclip = quirk && cls;
                const uint16_t* lut = slut + 128 * cls;
                uint32_t odd[FP];
                const int lanes = PER * st.z;
                if (NVX) {
                    row<KIND, (NVX ? NVX : 1), FP, PER, false>(R, app, msg, lanes, i, h, rec, 0, 0, noclip, lut, odd);
                } else {
                    const int lgs = (st.w >> 8) & 0xff;
                    const int left = (PER * st.z) - (i & ~31);
                    const unsigned m = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
                    switch (st.w & 0xff) {
                    case 1: row<KIND, 1, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    case 2: row<KIND, 2, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    case 3: row<KIND, 3, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    case 4: row<KIND, 4, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    case 5: row<KIND, 5, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    case 6: row<KIND, 6, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    case 7: row<KIND, 7, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    default: row<KIND, 8, FP, PER, true>(R, app, msg, lanes, i, h, rec, lgs, m, noclip, lut, odd); break;
                    }
                }
                if (KIND == KIND_2NMS) {
#pragma unroll
                    for (int p = 0; p < FP; p++) odd_any |= odd[p];
                } else if (ET) {
                    if (NVX || (k & ((1 << ((st.w >> 8) & 0xff)) - 1)) == 0) {
#pragma unroll
                        for (int p = 0; p < FP; p++) cnt[p] = h2::add(cnt[p], odd[p] | h2::ONE);
                        rows++;
                    }
                }
            }
            if (st.w & 0x10000) __syncthreads();
            st = nx;
            nx = nx2;
            rec = nrec;
            i = ni;
        }
        executed = it + 1;
        if (KIND == KIND_2NMS) {
            if (it >= 1 && !__syncthreads_or(odd_any != 0)) break;
        } else if (ET == 1) {
            unsigned odd = 0;
#pragma unroll
            for (int p = 0; p < FP; p++) odd += h2::odd_count(cnt[p], rows);
            if (odd_rows_within_slack(J, odd, it, s_odd) && !__syncthreads_or(odd_checks(L, app) != 0)) {
                passed = true;
                break;
            }
        } else if (ET == 2) {
            uint32_t oc[2] = {0, 0};  // odd rows of frames 0, 1 and 2, 3 in 16-bit halves
#pragma unroll
            for (int p = 0; p < FP; p++) {
                const __half2 c = *reinterpret_cast<const __half2*>(&cnt[p]);
                const uint32_t lo = (uint32_t)(rows - __half2int_rn(__low2half(c))) >> 1;
                const uint32_t hi = (uint32_t)(rows - __half2int_rn(__high2half(c))) >> 1;
                const uint32_t w = lo | hi << 16;
                if (FP == 2)
                    oc[p] = w;
                else if (threadIdx.x & 1)
                    oc[1] = w;
                else
                    oc[0] = w;
            }
            const uint2 t = odd_rows_total_lanes(oc[0], oc[1], it, s_odd);
            const unsigned n4[4] = {t.x & 0xffffu, t.x >> 16, t.y & 0xffffu, t.y >> 16};
            unsigned gate = 0;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (((live >> k) & 1u) && n4[k] <= J.early_slack) gate |= 1u << k;
            if (gate) {
                const uint32_t bad = odd_checks(L, app);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (((gate >> k) & 1u) && __syncthreads_or((bad >> (8 * k)) & 0xffu)) gate &= ~(1u << k);
                if (gate) {
                    write_hard(P, J, g, app, (int)gate);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if ((gate >> k) & 1u) its[k] = it + 1;
                    live &= ~gate;
                    if (!live) break;
                    __syncthreads();  // write_hard read the APP that the next iteration updates
                }
            }
        }
    }

    if (ET == 2) {
        if (live) write_hard(P, J, g, app, (int)live);
        if (J.iters_out && threadIdx.x == 0)
            for (int k = 0; k < 4; k++) J.iters_out[4 * (g - J.word0) + k] = ((live >> k) & 1u) ? executed : its[k];
        if (J.synd_out) {
            if (threadIdx.x == 0)
                for (int k = 0; k < 4; k++)
                    if (!((live >> k) & 1u)) J.synd_out[4 * (g - J.word0) + k] = 1;
            if (live) write_syndrome_flags(J, 4 * (g - J.word0), odd_checks(L, app), (int)live);
        }
        return;
    }
    const int kmask = HALF ? 3 << (2 * half) : 0xF;
    write_hard(P, J, g, app, kmask);
    if (J.iters_out && threadIdx.x == 0 && half == 0) J.iters_out[g - J.word0] = executed;
    if (J.synd_out) write_syndrome_flags(J, 4 * (g - J.word0), passed ? 0u : odd_checks(L, app), kmask);
    if (J.app_out) {
        // two bytes (frames) at a time
        uint16_t* ao = reinterpret_cast<uint16_t*>(J.app_out);
        for (int v = threadIdx.x; v < P.n; v += blockDim.x)
            for (int p = HALF ? half : 0; p < (HALF ? half + 1 : 2); p++)
                ao[2 * ((long long)v * J.total_words + g) + p] = reinterpret_cast<const uint16_t*>(app)[2 * v + p] ^ 0x7f7fu;
    }
    if (J.msg_out) {
        uint16_t* mo = reinterpret_cast<uint16_t*>(J.msg_out);
        for (int s = 0; s < L.nstep; s++) {
            const int4 t = __ldg(steps + s);
            const int nv = t.w & 0xff, lanes = PER * t.z;
            for (int x = threadIdx.x; x < t.z * 8; x += blockDim.x) {
                const int k = x >> 3, j = x & 7;
                if (j >= nv - (int)((__ldg(L.rec + t.x + k).x >> 1) & 1)) continue;
                for (int p = HALF ? half : 0; p < (HALF ? half + 1 : 2); p++) {
                    // pair p's bytes of edge j in the list of its lane, in its 16-, 8-, 4- or 2-byte part
                    const int l = PER == 2 ? 2 * k + p : k, eb = 2 * FP, bytes = nv * eb, b = j * eb + (FP == 2 ? 2 * p : 0);
                    int base = 0, part = 16;
                    while (base + part > bytes || b >= base + part) {
                        if (base + part <= bytes) base += part;
                        else part >>= 1;
                    }
                    const uint8_t* m = reinterpret_cast<const uint8_t*>(msgs + t.y + base * lanes + part * l + (b - base));
                    const uint32_t w = (uint8_t)(128 - (int)m[0]) | (uint32_t)(uint8_t)(128 - (int)m[1]) << 8;
                    mo[2 * ((long long)L.edge[8 * (t.x + k) + j] * J.total_words + g) + p] = (uint16_t)w;
                }
            }
        }
    }
}

template <int KIND, int NVX, int FP, int ET>
__global__ void __launch_bounds__(512) decode_level_bytes_kernel(const Plan P, const LevelPlan L, const Job J)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_odd[4];
    decode_word_bytes<KIND, NVX, FP, ET>(P, L, J, J.word0 + blockIdx.x, reinterpret_cast<char*>(smem_raw), s_odd);
}

// One frame pair per CTA (blockIdx.x = 2 * (g - word0) + half)
template <int KIND, int NVX>
__global__ void __launch_bounds__(512) decode_level_half_bytes_kernel(const Plan P, const LevelPlan L, const Job J)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_odd[4];
    decode_word_bytes<KIND, NVX, 1, 0, true>(P, L, J, J.word0 + (blockIdx.x >> 1), reinterpret_cast<char*>(smem_raw), s_odd,
                                             blockIdx.x & 1);
}

}  // namespace ldpc
