#include "kernels_level.cuh"

namespace ldpc {
extern const void* const level_kernels_f1_e0[5][3];
const void* const level_kernels_f1_e0[5][3] = {LDPC_LEVEL_ROWS(1, 0),
    LDPC_LEVEL_ROW(KIND_2NMS, 1, 0)};
}  // namespace ldpc
