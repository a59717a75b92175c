#include "kernels_level.cuh"

namespace ldpc {
extern const void* const level_kernels_f1_e1[4][3];
const void* const level_kernels_f1_e1[4][3] = {LDPC_LEVEL_ROWS(1, 1)};
}  // namespace ldpc
