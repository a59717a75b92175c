// Instantiations of decode_level_bytes_kernel: one unit per frame pairs per thread (FP) and early
// stop (ET), [kind: MS, OMS, NMS, LEARNED, 2NMS (fixed iterations only)][edges per row: any, 6, 7].
#pragma once
#include "level_kernel.cuh"

#define LDPC_LEVEL_ROW(KIND, FP, ET)                                                                       \
    {(const void*)decode_level_bytes_kernel<KIND, 0, FP, ET>, (const void*)decode_level_bytes_kernel<KIND, 6, FP, ET>, \
     (const void*)decode_level_bytes_kernel<KIND, 7, FP, ET>}
#define LDPC_LEVEL_ROWS(FP, ET)                                                                  \
    LDPC_LEVEL_ROW(KIND_MS, FP, ET), LDPC_LEVEL_ROW(KIND_OMS, FP, ET), LDPC_LEVEL_ROW(KIND_NMS, FP, ET), \
        LDPC_LEVEL_ROW(KIND_LEARNED, FP, ET)
