#include "kernels_level.cuh"

namespace ldpc {
extern const void* const level_kernels_f2_e0[5][3];
const void* const level_kernels_f2_e0[5][3] = {LDPC_LEVEL_ROWS(2, 0),
    LDPC_LEVEL_ROW(KIND_2NMS, 2, 0)};

#define LDPC_LEVEL_DECL(F, E) extern const void* const level_kernels_f##F##_e##E[][3];
LDPC_LEVEL_DECL(1, 0) LDPC_LEVEL_DECL(1, 1) LDPC_LEVEL_DECL(1, 2) LDPC_LEVEL_DECL(2, 0) LDPC_LEVEL_DECL(2, 1) LDPC_LEVEL_DECL(2, 2)

const void* kernel_table_level(int kind, int nv, int fp, int et)
{
    const int row = kind == KIND_LEARNED ? 3 : (kind == KIND_2NMS ? 4 : kind), col = nv == 6 ? 1 : (nv == 7 ? 2 : 0);
    if (kind == KIND_2NMS && et != 0) return nullptr;
    const void* const(*t)[3] = fp == 1 ? (et == 0 ? level_kernels_f1_e0 : (et == 1 ? level_kernels_f1_e1 : level_kernels_f1_e2))
                                       : (et == 0 ? level_kernels_f2_e0 : (et == 1 ? level_kernels_f2_e1 : level_kernels_f2_e2));
    return t[row][col];
}
}  // namespace ldpc
