// Kernel tables of the library: the address of each kernel instantiation,
// by measure, rows per thread and arithmetic mode.  The instantiations live
// in separate translation units (tsm_k_<family>_<mode>.cu), one per kernel
// family and mode, so that they compile in parallel; tsm_capi.cu launches
// them through these addresses.  Every function returns nullptr for an
// unsupported combination (rows per thread other than 4, 8, 16; the
// scheduler: 4, 8).
#pragma once

namespace tsm_k {

// dp_pairs_kernel / dp_matrix_kernel / dp_wave_kernel<M, R, EXACT>, M = TSM_DTW .. TSM_DFRECHET
// (dp_matrix: not EDR and LCSS)
const void* dp_pairs(int measure, int R, bool exact);
const void* dp_matrix(int measure, int R, bool exact);
const void* dp_wave(int measure, int R, bool exact);
// dp_matrix_lane_kernel<M, 8, EXACT>, M = TSM_DTW or TSM_DFRECHET
const void* dp_matrix_lane(int measure, bool exact);
const void* dp_matrix_lane_fast(int measure);
// bits_matrix_kernel<M, FEW>, M = TSM_EDR or TSM_LCSS
const void* bits_matrix(int measure, bool few);
// hausdorff_matrix_kernel (matrix) or hausdorff_pairs_kernel, and hausdorff_wave_kernel <R, EXACT>
const void* haus(bool matrix, int R, bool exact);
const void* haus_wave(int R, bool exact);
// hausdorff_pruned_matrix_kernel or (longs) hausdorff_long_matrix_kernel <QB, EXACT>, QB = 1 or 4, and
// hausdorff_pruned_pairs_kernel<TEAM, EXACT>
const void* haus_pruned_matrix(int QB, bool longs, bool exact);
const void* haus_pruned_pairs(bool team, bool exact);
// dp_sched_kernel<R, EXACT>
const void* sched(int R, bool exact);

// the default-mode halves (tsm_k_<family>_fast.cu)
const void* dp_pairs_fast(int measure, int R);
const void* dp_matrix_fast(int measure, int R);
const void* dp_wave_fast(int measure, int R);
const void* sched_fast(int R);

}  // namespace tsm_k
