// The persistent batch kernel with byte storage and fp16x2 arithmetic (level_kernel.cuh), the
// LDPC_PACK_SIMD4 one for codes that have that schedule.  Short irregular codes of rates 1/2 to
// 5/6, 50 000 words, early stop, at most 20 iterations: 40.5 ms with per-byte SIMD and rows of up
// to 32 unrolled edges, 6.3 ms here (rows over 1, 2 or 4 lanes of at most 8 edges).
//
// What bounds it: the latency of the steps, so the words that are resident count.  The record of
// the code and its job lie in shared memory: as local copies they took 128 to 151 registers a
// thread and 3 or 4 CTAs of 128 threads fitted a multiprocessor; with 96 registers 5 do.  us
// before and after: the above 6890 / 6256; the same codes, 300 words 278 / 259; each frame
// stopping on its own, 20 000 words 4782 / 3451; 20 fixed iterations, 20 000 words 4130 / 3959.
// The row update spills at 96 registers: 44 to 60 bytes without the early stop, 72 to 80 with it, 116 to
// 124 with the stop per frame (148 to 280 with 72 registers).  Without the early stop the schedule's
// pointers are better kept in registers (3959; from shared memory 4152), with it in shared memory
// (6256; in registers 6357).
#include "batch_kernel.cuh"

namespace ldpc {

template <int KIND, int ET>
__global__ void __launch_bounds__(320, 2) decode_batch_bytes_kernel(const BatchCode* __restrict__ codes, int n_codes,
                                                                    unsigned long long* counter, long long total,
                                                                    const __grid_constant__ Job base)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_odd[4];
    __shared__ long long s_item;
    __shared__ int s_code;  // the code that s_bc and s_job are of (thread 0)
    __shared__ __align__(16) unsigned char s_raw[sizeof(BatchCode)];  // (its members have initialisers)
    BatchCode& s_bc = *reinterpret_cast<BatchCode*>(s_raw);
    __shared__ Job s_job;
    if (threadIdx.x == 0) s_code = -1;
    for (;;) {
        if (threadIdx.x == 0) {
            const long long item = (long long)atomicAdd(counter, 1ull);
            s_item = item;
            if (item < total) {
                const int c = batch_code_of(codes, n_codes, item);
                if (c != s_code) {
                    s_code = c;
                    s_bc = codes[c];
                    batch_job(s_bc, base, s_job);
                }
            }
        }
        __syncthreads();
        const long long item = s_item;
        if (item >= total) break;  // uniform
        char* smem = reinterpret_cast<char*>(smem_raw);
        if (ET) {
            decode_word_bytes<KIND, 0, 2, ET>(s_bc.plan, s_bc.lplan, s_job, item - s_bc.first_item, smem, s_odd);
        } else {
            const LevelPlan L = s_bc.lplan;
            decode_word_bytes<KIND, 0, 2, ET>(s_bc.plan, L, s_job, item - s_bc.first_item, smem, s_odd);
        }
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
