// dp_matrix_kernel in default mode (hardware sqrt and reciprocal approximations)
// (table: tsm_kernels.h).
#include "tsm_tile.cuh"
#include "tsm_pick.cuh"

namespace tsm_k {

const void* dp_matrix_lane_fast(int measure) {
    return measure == TSM_DTW ? (const void*)&tsm::dp_matrix_lane_kernel<tsm::DTW, 8, false>
                              : (const void*)&tsm::dp_matrix_lane_kernel<tsm::DFRECHET, 8, false>;
}

const void* dp_matrix_fast(int measure, int R) {
    TSM_DP_MATRIX_TABLE(tsm::dp_matrix_kernel, false, measure, R)
}

}  // namespace tsm_k
