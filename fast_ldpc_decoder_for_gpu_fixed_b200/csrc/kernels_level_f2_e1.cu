#include "kernels_level.cuh"

namespace ldpc {
extern const void* const level_kernels_f2_e1[4][3];
const void* const level_kernels_f2_e1[4][3] = {LDPC_LEVEL_ROWS(2, 1)};
}  // namespace ldpc
