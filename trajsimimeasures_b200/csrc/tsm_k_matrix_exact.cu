// dp_matrix_kernel in exact mode (IEEE sqrt and reciprocal), and the table's entry point
// (tsm_kernels.h).
#include "tsm_tile.cuh"
#include "tsm_pick.cuh"

namespace tsm_k {

const void* dp_matrix_lane(int measure, bool exact) {
    if (!exact) return dp_matrix_lane_fast(measure);
    return measure == TSM_DTW ? (const void*)&tsm::dp_matrix_lane_kernel<tsm::DTW, 8, true>
                              : (const void*)&tsm::dp_matrix_lane_kernel<tsm::DFRECHET, 8, true>;
}

const void* dp_matrix(int measure, int R, bool exact) {
    if (!exact) return dp_matrix_fast(measure, R);
    TSM_DP_MATRIX_TABLE(tsm::dp_matrix_kernel, true, measure, R)
}

const void* bits_matrix(int measure, bool few) {
    if (few)
        return measure == TSM_EDR ? (const void*)&tsm::bits_matrix_kernel<tsm::EDR, true>
                                  : (const void*)&tsm::bits_matrix_kernel<tsm::LCSS, true>;
    return measure == TSM_EDR ? (const void*)&tsm::bits_matrix_kernel<tsm::EDR, false>
                              : (const void*)&tsm::bits_matrix_kernel<tsm::LCSS, false>;
}

}  // namespace tsm_k
