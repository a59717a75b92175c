// Training of the LDPC_LEARNED constants: FP32 forward and backward passes
// through the unrolled row-layered min-sum decoder, one CTA per frame.
//
// Forward model, per frame, iterations t = 0..T-1, rows in the decoder's level
// order, g = the row's class (degree group), j over the row's d edges, v_j its
// variables (the int8 decoders' semantics, with real-valued constants):
//   t_j   = clamp(a[v_j] - m_j, -128, 127)               (m_j = this edge's last message, 0 at t = 0)
//   u_j   = [t_j > 0]   (bit 1),  P = xor_j u_j
//   mag_j = min(|t_j|, 127);  min1 = mag_i1 <= min2 = mag_i2 <= the others
//   y(x)  = alpha[t][g] * x - beta[t][g]    or, with `quantized`, floor(alpha * x) - beta
//   c(x)  = clamp(y(x), 0, 31)
//   m_j   = (P ^ u_j ? +1 : -1) * (j == i1 ? c(min2) : c(min1))
//   a[v_j] = clamp(t_j + m_j, -128, 127)
// a starts as the channel LLRs in the int8 decoders' units.  With integer LLRs,
// alpha = s / 128 and integer beta, the quantized forward pass is exactly the
// LDPC_LEARNED int8 decoder (offsets beta, Q1.7 scales s): every value is an
// integer below 2^24, so FP32 holds it exactly.  Every forward operation is one
// IEEE FP32 operation rounded to nearest (no contraction into FMA), so a float32
// emulation reproduces the forward pass bit for bit.
//
// Loss, with w[t] the weight of iteration t (default: the last iteration only),
// a(t) the APP after iteration t, b the transmitted bits (a positive LLR means
// bit 1), kappa_f the frame's factor from the decoder's LLR units to natural
// log-likelihood ratios and S_f(t) = sum_v BCE(sigmoid(kappa_f a_v(t)), b_v):
//   bit loss   (LDPC_TRAIN_BIT_LOSS):   sum_t w[t] * mean_f S_f(t) / n
//   frame loss (LDPC_TRAIN_FRAME_LOSS): sum_t w[t] * mean_f (1 - exp(-S_f(t)))
// exp(-S_f) is the probability, under the soft output, that every bit of the
// frame is right, so the frame loss is a soft frame error rate.
//
// Backward: the reverse row sequence (levels in reverse order, the rows of a
// level in parallel, as in the forward pass).  Gradients are straight-through
// for min and sign (the argmins and signs found in the forward pass are held
// fixed), for the two saturations and for the floor; c's clamp passes the
// gradient only where 0 < y < 31.  The forward pass records {min1, min2,
// i1 | i2 << 8, sign bits} per row and iteration (16 bytes), and for weighted
// iterations before the last sigmoid - b of every variable (4 bytes) and S_f(t), in a
// caller-provided stash.
//
// The row updates are unrolled for each row's own degree, so that a row's values stay in
// registers: with loops over the degree they went through local memory, and the kernel waited
// on that (1.44 G warp instructions at 0.44 per cycle).  Unrolled for the largest degree of a class
// (8, 16, 32) and predicated, a row also waits for the edges that it does not have: us of a forward
// and backward pass, 600 frames, 5 iterations, with loops / by class / by degree: 1200x600 (degrees
// 8 and 9) 4772 / 7164 / 3173; 816x408 (10) 1003 / 1085 / 570; 2048x384 (32) 987 / 1181 / 521;
// 1944x972 (7 and 8) 384 / 209 / 170; 4000x2000 (6) 949 / 362 / 361.  Degrees above 16 spill beside 128
// registers (476 bytes), which costs less than reading their columns twice (2048x384: 574).  sigmoid - b comes from the forward
// pass's exp(-|z|) and is kept, so the backward pass evaluates no exponential.
// N = 4096 QC code, 2048 frames, 10 iterations, every iteration weighted, forward and backward,
// B200: 2.97 ms before, 1.15 ms now; its stash (0.67 GB) and sigmoids (0.30 GB), written and
// read once, take 0.3 ms of that.  What bounds it (592 frames, counters): issue slots 58 % and the ALU pipe 57 %
// busy with 4.8 warps a scheduler (registers and shared memory both allow 3 CTAs of 8 warps), DRAM 13 %;
// the rest is latency, of the columns' and the stash's loads first, with too few warps to hide it.
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "../../include/ldpc_b200.h"
#include "decode_kernel.cuh"

namespace ldpc {

struct TrainArgs {
    const float* llr;      // [frames][n]
    const uint8_t* bits;   // [frames][n] transmitted bits, or null for the all-zero codeword
    const float* kappa;    // [frames]
    const float* alpha;    // [T][2]
    const float* beta;     // [T][2]
    float* grad_alpha;     // [T][2] accumulated
    float* grad_beta;      // [T][2] accumulated
    float* loss;           // [1] accumulated
    uint4* stash;          // [frames][T][m]
    float* stash_app;      // [frames][T][n]: sigmoid(kappa a) - b
    float* stash_s;        // [frames][T]
    const float* weights;  // [T] loss weight per iteration, or null (last only)
    float* app_out;        // [frames][n] final soft output, or null
    int T;
    int quantized;
    int frame_loss;
    int backward;
    float inv_frames;      // 1 / frames
    float inv_n;           // 1 / n
};

__device__ __forceinline__ float warp_sum(float x)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// sum over the CTA (blockDim.x a multiple of 32, at most 256), returned to every thread
__device__ __forceinline__ float block_sum(float x, float* scratch)
{
    x = warp_sum(x);
    __syncthreads();  // scratch may still be read from a previous call
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = x;
    __syncthreads();
    float s = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += scratch[w];
    return s;
}

__device__ __forceinline__ float pre_mag(float al, float be, float x, int quantized)
{
    const float p = __fmul_rn(al, x);
    return __fsub_rn(quantized ? floorf(p) : p, be);
}

// BCE(sigmoid(z), b) = softplus(z) - b z and, in grad, its derivative sigmoid(z) - b: with
// e = exp(-|z|), 1 / (1 + e) or e / (1 + e) with the sign of b, without cancellation
__device__ __forceinline__ float bce(float z, bool b, float& grad)
{
    const float e = expf(-fabsf(z));
    const float g = ((z >= 0.f) == b ? e : 1.f) / (1.f + e);
    grad = b ? -g : g;
    return fmaxf(z, 0.f) + log1pf(e) - (b ? z : 0.f);
}

__device__ __forceinline__ float iter_weight(const TrainArgs& A, int t)
{
    return A.weights ? A.weights[t] : (t == A.T - 1 ? 1.f : 0.f);
}

// the loss term of iteration t for this frame from S = S_f(t), and the factor
// that multiplies kappa * (sigmoid - b) in its gradient
__device__ __forceinline__ float term_loss(const TrainArgs& A, float w, float S)
{
    return A.frame_loss ? w * (1.f - expf(-S)) * A.inv_frames : w * S * A.inv_n * A.inv_frames;
}
__device__ __forceinline__ float term_grad(const TrainArgs& A, float w, float S)
{
    return A.frame_loss ? w * expf(-S) * A.inv_frames : w * A.inv_n * A.inv_frames;
}

// The frame's loss sum S_f over its variables (one part per thread) from the APP in shared
// memory, and sigmoid - b into g (null: not wanted; may be a itself).  VEC: four variables at a
// time (n a multiple of 4, the buffers aligned for it).
template <bool VEC>
__device__ __forceinline__ float frame_part(const TrainArgs& A, int n, long long f, float kap, const float* a, float* g)
{
    float part = 0.f;
    if (VEC) {
        for (int q = threadIdx.x; q < (n >> 2); q += blockDim.x) {
            const float4 x = reinterpret_cast<const float4*>(a)[q];
            const uchar4 b = A.bits ? __ldg(reinterpret_cast<const uchar4*>(A.bits + f * n) + q) : make_uchar4(0, 0, 0, 0);
            float4 d;
            part += bce(kap * x.x, b.x, d.x);
            part += bce(kap * x.y, b.y, d.y);
            part += bce(kap * x.z, b.z, d.z);
            part += bce(kap * x.w, b.w, d.w);
            if (g) reinterpret_cast<float4*>(g)[q] = d;
        }
    } else {
        for (int v = threadIdx.x; v < n; v += blockDim.x) {
            float d;
            part += bce(kap * a[v], A.bits ? A.bits[f * n + v] != 0 : false, d);
            if (g) g[v] = d;
        }
    }
    return part;
}

// What the backward pass needs of a row's update: its minima, their edges and the signs.
struct RowMinima {
    float m1, m2;
    int i1, i2;
    uint32_t pos;
};

// The update of a row of D edges.  c: its first column in the code's table, the others m entries apart;
// msg: its messages, likewise.
template <int D>
__device__ __forceinline__ RowMinima row_forward(const uint16_t* c, int m, float* a, float* msg, float al, float be, int quantized)
{
    RowMinima R{127.f, 127.f, 0, 1, 0u};
    float tv[D];
    int vo[D];
#pragma unroll
    for (int j = 0; j < D; j++) vo[j] = __ldg(c + j * m);
#pragma unroll
    for (int j = 0; j < D; j++) tv[j] = fminf(fmaxf(__fsub_rn(a[vo[j]], msg[j * m]), -128.f), 127.f);
#pragma unroll
    for (int j = 0; j < D; j++) {
        const float ax = fminf(fabsf(tv[j]), 127.f);
        R.pos |= (tv[j] > 0.f ? 1u : 0u) << j;
        const bool lt1 = ax < R.m1, lt2 = ax < R.m2;
        R.i2 = lt1 ? R.i1 : (lt2 ? j : R.i2);
        R.i1 = lt1 ? j : R.i1;
        R.m2 = fminf(R.m2, fmaxf(R.m1, ax));
        R.m1 = fminf(R.m1, ax);
    }
    if (R.i2 == R.i1) R.i2 = R.i1 + 1 < D ? R.i1 + 1 : 0;  // all other magnitudes 127: any second edge
    const float c1 = fminf(fmaxf(pre_mag(al, be, R.m2, quantized), 0.f), 31.f);
    const float c2 = fminf(fmaxf(pre_mag(al, be, R.m1, quantized), 0.f), 31.f);
    const uint32_t neg = (__popc(R.pos) & 1) ? R.pos : ~R.pos;  // bit j: the message of edge j is negative
#pragma unroll
    for (int j = 0; j < D; j++) {
        const float mag = j == R.i1 ? c1 : c2;
        const float mj = ((neg >> j) & 1) ? -mag : mag;
        msg[j * m] = mj;
        a[vo[j]] = fminf(fmaxf(__fadd_rn(tv[j], mj), -128.f), 127.f);
    }
    return R;
}

// The reverse of row_forward: a and msg hold the gradients of the APPs and of the messages after the row,
// then those before it.  Adds the row's gradients of alpha and beta to da and db.
template <int D>
__device__ __forceinline__ void row_backward(const uint16_t* c, int m, float* a, float* msg, const RowMinima& R, float al, float be,
                                             int quantized, float& da, float& db)
{
    const uint32_t neg = (__popc(R.pos) & 1) ? R.pos : ~R.pos;
    float gt[D];
    int vo[D];
#pragma unroll
    for (int j = 0; j < D; j++) vo[j] = __ldg(c + j * m);
    float gc1 = 0.f, gc2 = 0.f;
#pragma unroll
    for (int j = 0; j < D; j++) {
        gt[j] = a[vo[j]];                         // d/d a[v] after this row
        const float gm = gt[j] + msg[j * m];      // d/d m_j: the APP and the next iteration
        const float s = ((neg >> j) & 1) ? -gm : gm;
        gc1 = j == R.i1 ? s : gc1;
        gc2 += j == R.i1 ? 0.f : s;
    }
    float gm1 = 0.f, gm2 = 0.f;
    const float y1 = pre_mag(al, be, R.m2, quantized), y2 = pre_mag(al, be, R.m1, quantized);
    if (y1 > 0.f && y1 < 31.f) {
        da += R.m2 * gc1;
        db -= gc1;
        gm2 = al * gc1;
    }
    if (y2 > 0.f && y2 < 31.f) {
        da += R.m1 * gc2;
        db -= gc2;
        gm1 = al * gc2;
    }
    // min1 = |t_i1|, min2 = |t_i2|; d|t|/dt = +1 for t > 0, -1 otherwise
    gm1 = ((R.pos >> R.i1) & 1) ? gm1 : -gm1;
    gm2 = ((R.pos >> R.i2) & 1) ? gm2 : -gm2;
#pragma unroll
    for (int j = 0; j < D; j++) {
        const float x = gt[j] + (j == R.i1 ? gm1 : (j == R.i2 ? gm2 : 0.f));
        a[vo[j]] = x;     // d/d a[v] before this row
        msg[j * m] = -x;  // d/d (this edge's message of iteration t-1)
    }
}

// Calls f with the degree d (1 to MOST) as a compile-time constant.
template <int MOST, int D = 1, class F>
__device__ __forceinline__ void with_degree(int d, F f)
{
    if constexpr (D == MOST) {
        f(std::integral_constant<int, D>());
    } else {
        if (d == D) f(std::integral_constant<int, D>());
        else with_degree<MOST, D + 1>(d, f);
    }
}

// DT: the largest degree; UNIFORM: every row has it
template <int DT, bool UNIFORM, bool VEC>
__global__ void __launch_bounds__(256, DT <= 8 ? 3 : 2) train_kernel(const Plan P, const TrainArgs A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* a = reinterpret_cast<float*>(smem_raw);    // APP, then its gradient
    float* msg = a + P.npad;                          // messages [dmax][m], then their gradients
    __shared__ float gpar[4 * LDPC_LEARNED_MAX_ITERS];  // [t][g][d alpha, d beta]
    __shared__ float scratch[8];
    const long long f = blockIdx.x;
    const int T = A.T;

    for (int i = threadIdx.x; i < 4 * LDPC_LEARNED_MAX_ITERS; i += blockDim.x) gpar[i] = 0.f;
    if (VEC)
        for (int q = threadIdx.x; q < (P.n >> 2); q += blockDim.x)
            reinterpret_cast<float4*>(a)[q] = __ldg(reinterpret_cast<const float4*>(A.llr + f * P.n) + q);
    else
        for (int v = threadIdx.x; v < P.n; v += blockDim.x) a[v] = A.llr[f * P.n + v];
    for (int i = threadIdx.x; i < P.dmax * P.m; i += blockDim.x) msg[i] = 0.f;
    __syncthreads();

    const float kap = A.kappa[f];
    float floss = 0.f;  // this frame's loss (thread 0)

    // ---------------- forward ----------------
    for (int t = 0; t < T; t++) {
        const float al0 = A.alpha[2 * t], al1 = A.alpha[2 * t + 1], be0 = A.beta[2 * t], be1 = A.beta[2 * t + 1];
        for (int l = 0; l < P.nlevels; l++) {
            const int2 lv = __ldg(P.levels + l);
            for (int r = lv.x + threadIdx.x; r < lv.x + lv.y; r += blockDim.x) {
                const int d = UNIFORM ? DT : __ldg(P.rowdeg + r), g = __ldg(P.rowcls + r);
                const float al = g ? al1 : al0, be = g ? be1 : be0;
                auto row = [&](auto D) {
                    const RowMinima R = row_forward<D.value>(P.cols + r, P.m, a, msg + r, al, be, A.quantized);
                    if (A.backward)
                        A.stash[((size_t)f * T + t) * P.m + r] =
                            make_uint4(__float_as_uint(R.m1), __float_as_uint(R.m2), (uint32_t)(R.i1 | (R.i2 << 8)), R.pos);
                };
                if constexpr (UNIFORM) row(std::integral_constant<int, DT>());
                else with_degree<DT>(d, row);
            }
            __syncthreads();
        }
        // intermediate loss terms: their gradients' sigmoids and S_f(t) are kept for the backward pass
        const float w = iter_weight(A, t);
        if (t < T - 1 && w != 0.f) {
            const float part =
                frame_part<VEC>(A, P.n, f, kap, a, A.backward ? A.stash_app + ((size_t)f * T + t) * P.n : nullptr);
            const float S = block_sum(part, scratch);  // also orders the reads of a before iteration t+1
            floss += term_loss(A, w, S);
            if (A.backward && threadIdx.x == 0) A.stash_s[(size_t)f * T + t] = S;
        }
    }

    // ---------------- final loss term and its gradient ----------------
    {
        if (A.app_out)
            for (int v = threadIdx.x; v < P.n; v += blockDim.x) A.app_out[f * P.n + v] = a[v];
        if (A.app_out) __syncthreads();
        const float w = iter_weight(A, T - 1);
        const float S = block_sum(frame_part<VEC>(A, P.n, f, kap, a, A.backward ? a : nullptr), scratch);
        floss += term_loss(A, w, S);
        if (threadIdx.x == 0) atomicAdd(A.loss, floss);
        if (!A.backward) return;
        const float coef = term_grad(A, w, S) * kap;
        for (int v = threadIdx.x; v < P.n; v += blockDim.x) a[v] *= coef;
        for (int i = threadIdx.x; i < P.dmax * P.m; i += blockDim.x) msg[i] = 0.f;
        __syncthreads();
    }

    // ---------------- backward ----------------
    for (int t = T - 1; t >= 0; t--) {
        float ga0 = 0.f, ga1 = 0.f, gb0 = 0.f, gb1 = 0.f;
        const float w = iter_weight(A, t);
        if (t < T - 1 && w != 0.f) {  // the loss term on the APP after iteration t
            const float* keep = A.stash_app + ((size_t)f * T + t) * P.n;
            const float coef = term_grad(A, w, A.stash_s[(size_t)f * T + t]) * kap;
            if (VEC) {
                for (int q = threadIdx.x; q < (P.n >> 2); q += blockDim.x) {
                    const float4 k = reinterpret_cast<const float4*>(keep)[q];
                    float4 x = reinterpret_cast<float4*>(a)[q];
                    x.x += coef * k.x, x.y += coef * k.y, x.z += coef * k.z, x.w += coef * k.w;
                    reinterpret_cast<float4*>(a)[q] = x;
                }
            } else {
                for (int v = threadIdx.x; v < P.n; v += blockDim.x) a[v] += coef * keep[v];
            }
            __syncthreads();
        }
        const float al0 = A.alpha[2 * t], al1 = A.alpha[2 * t + 1], be0 = A.beta[2 * t], be1 = A.beta[2 * t + 1];
        for (int l = P.nlevels - 1; l >= 0; l--) {
            const int2 lv = __ldg(P.levels + l);
            for (int r = lv.x + threadIdx.x; r < lv.x + lv.y; r += blockDim.x) {
                const int d = UNIFORM ? DT : __ldg(P.rowdeg + r), g = __ldg(P.rowcls + r);
                const uint4 st = A.stash[((size_t)f * T + t) * P.m + r];
                const float al = g ? al1 : al0, be = g ? be1 : be0;
                const RowMinima R{__uint_as_float(st.x), __uint_as_float(st.y), (int)(st.z & 0xff), (int)((st.z >> 8) & 0xff), st.w};
                float da = 0.f, db = 0.f;
                auto row = [&](auto D) {
                    row_backward<D.value>(P.cols + r, P.m, a, msg + r, R, al, be, A.quantized, da, db);
                };
                if constexpr (UNIFORM) row(std::integral_constant<int, DT>());
                else with_degree<DT>(d, row);
                ga0 += g ? 0.f : da, gb0 += g ? 0.f : db;
                ga1 += g ? da : 0.f, gb1 += g ? db : 0.f;
            }
            __syncthreads();
        }
        const float x[4] = {warp_sum(ga0), warp_sum(gb0), warp_sum(ga1), warp_sum(gb1)};
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int i = 0; i < 4; i++) atomicAdd(&gpar[4 * t + i], x[i]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * T; i += blockDim.x) {
        atomicAdd(A.grad_alpha + i, gpar[2 * i + 0]);
        atomicAdd(A.grad_beta + i, gpar[2 * i + 1]);
    }
}

template <bool VEC>
static const void* train_kernel_for(int dmax, bool uniform)
{
    if (uniform && dmax == 6) return (const void*)train_kernel<6, true, VEC>;
    if (uniform && dmax == 7) return (const void*)train_kernel<7, true, VEC>;
    if (dmax <= 8) return (const void*)train_kernel<8, false, VEC>;
    if (dmax <= 16) return (const void*)train_kernel<16, false, VEC>;
    return (const void*)train_kernel<32, false, VEC>;
}

}  // namespace ldpc

using namespace ldpc;

int ldpc_internal_fail(int code, const char* msg);
int ldpc_internal_plan(const ldpc_decoder* dec, Plan* plan, int* threads, bool* uniform);
cudaError_t ldpc_internal_raise_smem(const void* fn, size_t bytes);

static size_t stash_rows(const Plan& P, size_t frames, int iters) { return frames * (size_t)iters * P.m * sizeof(uint4); }
static size_t stash_apps(const Plan& P, size_t frames, int iters) { return frames * (size_t)iters * P.n * sizeof(float); }

extern "C" size_t ldpc_train_stash_bytes(const ldpc_decoder* dec, size_t frames, int iters)
{
    Plan P;
    int threads = 0;
    bool uniform = false;
    if (!dec || iters < 1 || ldpc_internal_plan(dec, &P, &threads, &uniform)) return 0;
    return stash_rows(P, frames, iters) + stash_apps(P, frames, iters) + frames * (size_t)iters * sizeof(float);
}

extern "C" int ldpc_train_step(const ldpc_decoder* dec, const float* d_llr, const uint8_t* d_bits,
                               const float* d_kappa, size_t frames, int iters, int flags,
                               const float* d_alpha, const float* d_beta, const float* d_weights,
                               float* d_grad_alpha, float* d_grad_beta, float* d_loss, void* d_stash,
                               float* d_app_out, void* stream)
{
    if (!dec || !d_llr || !d_kappa || !d_alpha || !d_beta || !d_loss)
        return ldpc_internal_fail(LDPC_ERR_ARG, "ldpc_train_step: null pointer");
    if (flags & ~(LDPC_TRAIN_QUANTIZED | LDPC_TRAIN_FRAME_LOSS))
        return ldpc_internal_fail(LDPC_ERR_ARG, "ldpc_train_step: unknown flags");
    const bool backward = d_grad_alpha || d_grad_beta || d_stash;
    if (backward && !(d_grad_alpha && d_grad_beta && d_stash))
        return ldpc_internal_fail(LDPC_ERR_ARG, "ldpc_train_step: gradients need grad_alpha, grad_beta and stash");
    if (iters < 1 || iters > LDPC_LEARNED_MAX_ITERS)
        return ldpc_internal_fail(LDPC_ERR_ARG, "ldpc_train_step: iterations must be in [1, 32]");
    if (frames < 1 || frames > 0x7fffffffu) return ldpc_internal_fail(LDPC_ERR_SHAPE, "ldpc_train_step: frames");
    Plan P;
    int threads = 0;
    bool uniform = false;
    if (ldpc_internal_plan(dec, &P, &threads, &uniform))
        return ldpc_internal_fail(LDPC_ERR_ARG, "ldpc_train_step: decoder has no row schedule");
    if (P.dmax > 32 || P.dmax < 2)
        return ldpc_internal_fail(LDPC_ERR_UNSUPPORTED, "ldpc_train_step: row degrees must be in [2, 32]");
    const size_t smem = 4 * ((size_t)P.npad + (size_t)P.dmax * P.m);
    int dev = 0, smem_max = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem + 16 * LDPC_LEARNED_MAX_ITERS + 64 > (size_t)smem_max)
        return ldpc_internal_fail(LDPC_ERR_UNSUPPORTED,
                                  "ldpc_train_step: one frame's FP32 state does not fit in shared memory");
    TrainArgs A;
    A.llr = d_llr;
    A.bits = d_bits;
    A.kappa = d_kappa;
    A.alpha = d_alpha;
    A.beta = d_beta;
    A.grad_alpha = d_grad_alpha;
    A.grad_beta = d_grad_beta;
    A.loss = d_loss;
    char* sb = reinterpret_cast<char*>(d_stash);
    A.stash = reinterpret_cast<uint4*>(sb);
    A.stash_app = sb ? reinterpret_cast<float*>(sb + stash_rows(P, frames, iters)) : nullptr;
    A.stash_s = sb ? reinterpret_cast<float*>(sb + stash_rows(P, frames, iters) + stash_apps(P, frames, iters))
                   : nullptr;
    A.weights = d_weights;
    A.app_out = d_app_out;
    A.T = iters;
    A.quantized = (flags & LDPC_TRAIN_QUANTIZED) ? 1 : 0;
    A.frame_loss = (flags & LDPC_TRAIN_FRAME_LOSS) ? 1 : 0;
    A.backward = backward ? 1 : 0;
    A.inv_frames = (float)(1.0 / (double)frames);
    A.inv_n = (float)(1.0 / (double)P.n);
    auto aligned = [](const void* p, size_t to) { return ((uintptr_t)p & (to - 1)) == 0; };
    const bool vec = P.n % 4 == 0 && aligned(d_llr, 16) && aligned(d_bits, 4) && aligned(A.stash_app, 16);
    const void* fn = vec ? train_kernel_for<true>(P.dmax, uniform) : train_kernel_for<false>(P.dmax, uniform);
    cudaError_t e = ldpc_internal_raise_smem(fn, smem);
    if (e == cudaSuccess) {
        void* args[] = {(void*)&P, (void*)&A};
        e = cudaLaunchKernel(fn, dim3((unsigned)frames), dim3(threads), args, smem, (cudaStream_t)stream);
    }
    return e == cudaSuccess ? LDPC_OK : ldpc_internal_fail(LDPC_ERR_CUDA, cudaGetErrorString(e));
}
