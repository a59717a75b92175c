// The persistent batch kernel with byte storage and fp16x2 arithmetic (level_kernel.cuh), the
// LDPC_PACK_SIMD4 one for codes that have that schedule.  Short irregular codes of rates 1/2 to
// 5/6, 50 000 words, early stop, at most 20 iterations: 40.5 ms with per-byte SIMD and rows of up
// to 32 unrolled edges, 6.8 ms here (rows over 1, 2 or 4 lanes of at most 8 edges).
#include "batch_kernel.cuh"

namespace ldpc {

template <int KIND, int ET>
__global__ void __launch_bounds__(256) decode_batch_bytes_kernel(const BatchCode* __restrict__ codes, int n_codes,
                                                                 unsigned long long* counter, long long total, const Job base)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_odd[4];
    __shared__ long long s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = (long long)atomicAdd(counter, 1ull);
        __syncthreads();
        const long long item = s_item;
        if (item >= total) break;  // uniform
        Job J;
        const BatchCode& bc = batch_item(codes, n_codes, item, base, J);
        const Plan P = bc.plan;
        const LevelPlan L = bc.lplan;
        decode_word_bytes<KIND, 0, 2, ET>(P, L, J, item - bc.first_item, reinterpret_cast<char*>(smem_raw), s_odd);
        __syncthreads();  // shared memory and s_item are reused by the next item
    }
}

#define LDPC_BATCH_ROW(KIND)                                                                            \
    {(const void*)decode_batch_bytes_kernel<KIND, 0>, (const void*)decode_batch_bytes_kernel<KIND, 1>, \
     (const void*)decode_batch_bytes_kernel<KIND, 2>}

// [kind: MS, OMS, NMS, LEARNED][early stop: none, per word, per frame]
const void* kernel_table_batch_bytes(int kind, int et)
{
    static const void* table[4][3] = {LDPC_BATCH_ROW(KIND_MS), LDPC_BATCH_ROW(KIND_OMS), LDPC_BATCH_ROW(KIND_NMS),
                                      LDPC_BATCH_ROW(KIND_LEARNED)};
    if (kind == KIND_2NMS) return et == 0 ? (const void*)decode_batch_bytes_kernel<KIND_2NMS, 0> : nullptr;
    return table[kind == KIND_LEARNED ? 3 : kind][et];
}

}  // namespace ldpc
