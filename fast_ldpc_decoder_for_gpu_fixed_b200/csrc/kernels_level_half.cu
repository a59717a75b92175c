#include "kernels_level.cuh"

namespace ldpc {

#define LDPC_LEVEL_HALF(KIND)                                                                                  \
    {(const void*)decode_level_half_bytes_kernel<KIND, 0>, (const void*)decode_level_half_bytes_kernel<KIND, 6>, \
     (const void*)decode_level_half_bytes_kernel<KIND, 7>}

// [kind: MS, OMS, NMS][edges per row: any, 6, 7]
const void* kernel_table_level_half(int kind, int nv)
{
    static const void* table[3][3] = {LDPC_LEVEL_HALF(KIND_MS), LDPC_LEVEL_HALF(KIND_OMS), LDPC_LEVEL_HALF(KIND_NMS)};
    return kind < 0 || kind > KIND_NMS ? nullptr : table[kind][nv == 6 ? 1 : (nv == 7 ? 2 : 0)];
}

}  // namespace ldpc
