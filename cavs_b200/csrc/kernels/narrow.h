// The narrow levels of the fp32 Tree-LSTM as one persistent launch per direction (kernels/narrow_f32.cu).
#ifndef CAVS_B200_KERNELS_NARROW_H_
#define CAVS_B200_KERNELS_NARROW_H_

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace cavs_b200 {

// How a range of levels is cut over CTAs: col_groups x row_groups of them, w hidden units each.  w == 0: these sizes
// do not fit.  level_us: estimated time of a level of `rows` rows.
struct NarrowPlan {
  int w = 0, col_groups = 0, row_groups = 0, buffers = 0;
  size_t smem = 0;
  double level_us = 0.0;
};
NarrowPlan PlanNarrow(int H, int K, int rows, bool backward);

// Levels [level_begin, level_end) in ascending order; level_off: device copy of the level offsets.  Arrays as for the
// per-level launches (kernels/cell.h): S / HK, the saved gates [n_total, (3+K)H] and h|c of every row are written.
// barrier: a zeroed word; status: raised when a bounded wait expires.
struct NarrowForwardArgs {
  float *state, *gates, *S, *HK;
  const float *A, *U_iou, *U_f, *bias;
  const int32_t *child, *a_row, *level_off;   // child: state rows of the children
  unsigned* barrier;
  int* status;
  int n_total, level_begin, level_end, H;
  int w, col_groups, row_groups;              // from the plan
};
int LaunchNarrowForward(const NarrowPlan& plan, NarrowForwardArgs args, int K, cudaStream_t st);

// Levels [level_begin, level_end) in descending order: dA, ZF, and d(h|c) in the children's mailbox rows.  dz / Wc / C,
// dOut, child_state and dB_part as for LaunchCellBwd.
struct NarrowBackwardArgs {
  float *dA, *ZF, *mailbox, *dB_part;
  const float *dOut, *dz, *Wc, *gates, *state, *U_iou, *U_f;
  const int32_t *child, *child_state, *parent, *level_off;
  unsigned* barrier;
  int* status;
  int n_total, level_begin, level_end, H, C;
  int w, col_groups, row_groups, buffers;     // from the plan
};
int LaunchNarrowBackward(const NarrowPlan& plan, NarrowBackwardArgs args, int K, cudaStream_t st);

}  // namespace cavs_b200
#endif
