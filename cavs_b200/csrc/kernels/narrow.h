// The narrow levels of the Tree-LSTM as one persistent launch per direction (kernels/narrow_f32.cu, narrow_bf16.cu).
#ifndef CAVS_B200_KERNELS_NARROW_H_
#define CAVS_B200_KERNELS_NARROW_H_

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace cavs_b200 {

// How a range of levels is cut over CTAs: col_groups x row_groups of them, w hidden units each.  w == 0: these sizes
// do not fit.  level_us: what the bf16 plan was chosen by, an upper estimate of a level's time.
struct NarrowPlan {
  int w = 0, col_groups = 0, row_groups = 0, buffers = 0;
  size_t smem = 0;
  double level_us = 0.0;
};
NarrowPlan PlanNarrowF32(int H, int K, int rows, bool backward);
NarrowPlan PlanNarrowBf16(int H, int K, int rows, bool backward);
// Estimated microseconds of an fp32 level under a plan.
double NarrowLevelUsF32(const NarrowPlan& plan, int H, int K, int rows, bool backward);

// Levels [level_begin, level_end) in ascending order; level_off: device copy of the level offsets.  Arrays as for the
// per-level launches (kernels/cell.h): S / HK, the saved gates and h|c of every row are written.  A, S, HK and the
// weights are fp32, or bf16 with fp16 gates; i|o|u of row t at gates + t * pitch3, f_0.. at gates_f + t * pitch_f.
// barrier: a zeroed word; status: raised when a bounded wait expires; withhold: 1 keeps the
// grid barrier from ever completing (a test of its wait).
struct NarrowForwardArgs {
  float* state;
  void *gates, *gates_f, *S, *HK;
  const void *A, *U_iou, *U_f;
  const float* bias;
  const int32_t *child, *a_row, *level_off;   // child: state rows of the children
  unsigned* barrier;
  int* status;
  unsigned withhold;
  long long pitch3, pitch_f;
  int n_total, level_begin, level_end, H;
  int w, col_groups, row_groups, buffers;     // from the plan
};
int LaunchNarrowForwardF32(const NarrowPlan& plan, NarrowForwardArgs args, int K, cudaStream_t st);
int LaunchNarrowForwardBf16(const NarrowPlan& plan, NarrowForwardArgs args, int K, cudaStream_t st);

// Levels [level_begin, level_end) in descending order: dA, ZF, and d(h|c) in the children's mailbox rows.  dz / Wc / C,
// dOut, child_state and dB_part as for LaunchCellBwd.
struct NarrowBackwardArgs {
  void *dA, *ZF;
  float *mailbox, *dB_part;
  const void *gates, *gates_f, *U_iou, *U_f;
  const float *dOut, *dz, *Wc, *state;
  const int32_t *child, *child_state, *parent, *level_off;
  unsigned* barrier;
  int* status;
  unsigned withhold;
  long long pitch3, pitch_f;
  int n_total, level_begin, level_end, H, C;
  int w, col_groups, row_groups, buffers;     // from the plan
};
int LaunchNarrowBackwardF32(const NarrowPlan& plan, NarrowBackwardArgs args, int K, cudaStream_t st);
int LaunchNarrowBackwardBf16(const NarrowPlan& plan, NarrowBackwardArgs args, int K, cudaStream_t st);

}  // namespace cavs_b200
#endif
