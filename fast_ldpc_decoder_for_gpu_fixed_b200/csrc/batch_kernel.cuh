// The persistent batch kernels' record of one code and the choice of the next word.
#pragma once
#include "level_kernel.cuh"

namespace ldpc {

struct BatchCode {
    Plan plan;
    LevelPlan lplan;        // decode_batch_bytes_kernel's schedule
    const int8_t* llr;      // frame-major int8, 4 * words frames
    void* out;              // 0/1 bytes (or packed bits), frame-major
    int32_t* iters_out;     // [words] or null
    uint8_t* synd_out;      // [4 * words] per-frame syndrome flags or null
    long long words;
    long long first_item;   // items of the codes before this one
    int quirk;              // OMS first-iteration quirk (row classes of this code)
    int out_packed;
    int variant;            // this code's row-degree class: 0 <= 8, 1 <= 16, 2 <= 32
};

// The code of item `item` of the batch.
__device__ __forceinline__ int batch_code_of(const BatchCode* codes, int n_codes, long long item)
{
    int c = 0;
    while (c + 1 < n_codes && item >= codes[c + 1].first_item) c++;
    return c;
}

// J = the batch's job with the buffers of code bc.
__device__ __forceinline__ void batch_job(const BatchCode& bc, const Job& base, Job& J)
{
    J = base;
    J.llr = bc.llr;
    J.out = bc.out;
    J.out_packed = bc.out_packed;
    J.iters_out = bc.iters_out;
    J.synd_out = bc.synd_out;
    J.total_words = bc.words;
    J.word0 = 0;
    J.quirk = bc.quirk;
}

// The job of item `item` of the batch: its code's record, the word in that code.
__device__ __forceinline__ const BatchCode& batch_item(const BatchCode* codes, int n_codes, long long item, const Job& base,
                                                       Job& J)
{
    const BatchCode& bc = codes[batch_code_of(codes, n_codes, item)];
    batch_job(bc, base, J);
    return bc;
}

}  // namespace ldpc
