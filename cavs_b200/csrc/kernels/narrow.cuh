// What the persistent launches over narrow levels share in fp32 (narrow_f32.cu) and bf16 (narrow_bf16.cu): the grid
// barrier, the gate gradients of the backward pass, the cooperative launch.
#ifndef CAVS_B200_KERNELS_NARROW_CUH_
#define CAVS_B200_KERNELS_NARROW_CUH_

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "abi_common.h"
#include "kernels/bulk.cuh"
#include "kernels/cell.h"
#include "kernels/launch.h"
#include "kernels/narrow.h"

namespace cavs_b200 {
namespace narrow {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr size_t kMaxSmem = 226 * 1024;
constexpr unsigned kBarrierPolls = 1u << 19;   // about half a second

// The cell kernels' activations (kernels/cell.cu): libm-accurate for fp32, exp2-unit forms for bf16.
template <bool kFast>
__device__ __forceinline__ float Sigmoid(float x) { return kFast ? __fdividef(1.0f, 1.0f + __expf(-x)) : 1.0f / (1.0f + expf(-x)); }
template <bool kFast>
__device__ __forceinline__ float Tanh(float x) { return kFast ? 1.0f - __fdividef(2.0f, __expf(2.0f * x) + 1.0f) : tanhf(x); }

__device__ __forceinline__ float LoadCg(const float* p) { return __ldcg(p); }
__device__ __forceinline__ float LoadCg(const __half* p) { return __half2float(__ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p)))); }
__device__ __forceinline__ void StoreAs(float* p, float x) { *p = x; }
__device__ __forceinline__ void StoreAs(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }
__device__ __forceinline__ void StoreAs(__half* p, float x) { *p = __float2half_rn(x); }

// Grid barrier in two halves, so that requests for data that does not depend on it go out in between.  Arrival releases
// the CTA's writes (the red is cumulative over what __syncthreads ordered before it); the wait acquires the others', and
// returns false, *status raised, if they take too long.  All CTAs are resident: the launch is cooperative.
__device__ __forceinline__ void GridArrive(unsigned* counter) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
}
__device__ __forceinline__ bool GridWait(unsigned* counter, unsigned target, int* status) {
  __shared__ int s_ok;
  if (threadIdx.x == kThreads - 32) {   // a warp with few or no rows of its own to request
    int ok = 0;
    for (unsigned it = 0; it < kBarrierPolls; ++it) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if (v >= target) { ok = 1; break; }
    }
    if (!ok) atomicExch(status, 1);
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// The last phase waited for of each buffer, once more and bounded.  Out of line: it never runs, but a pass over 96 chains
// of two bf16 layers takes 2536 us with it inlined at the kernels' exits, 2530 so, 2517 without (and 2638 where the waits
// themselves went on waiting).
static __device__ __noinline__ void DrainRows(const uint64_t* bars, int buffers, uint32_t phases) {
  for (int buf = 0; buf < buffers; ++buf)
    for (uint32_t it = 0; it < (1u << 18); ++it) {
      uint32_t done;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(done) : "r"(bulk::SmemAddr(bars + buf)), "r"(((phases >> buf) & 1) ^ 1) : "memory");
      if (done) break;
    }
}

// Rows that arrive in shared memory by bulk copies, one mbarrier per buffer.  A row is one copy: with nearly all of an SM's
// memory given to shared memory, per-thread asynchronous copies have so little of L1 left to fly through that issuing
// 128 KB of them took 6.1 k clocks.  Sources were written by other SMs' ordinary stores before the grid barrier, hence the
// proxy fence of the issuing lanes.
template <int kBuffers>
struct BulkRows {
  uint64_t* bars;
  uint32_t phases = 0;
  bool ok = true;
  __device__ __forceinline__ void Init(uint64_t* shared, int arrivals) {   // followed by a __syncthreads of the caller
    bars = shared;
    if (threadIdx.x == 0) {
      for (int i = 0; i < kBuffers; ++i) bulk::MbarInit(bulk::SmemAddr(bars + i), arrivals);
      bulk::FenceMbarInit();
    }
  }
  // By one warp: lane r copies `bytes` from src (nullptr: nothing) to dst + r * pitch; one arrival.
  __device__ __forceinline__ void Copy(int buf, uint32_t dst, uint32_t pitch, const void* src, uint32_t bytes) {
    const int lane = threadIdx.x & 31;
    const unsigned live = __ballot_sync(0xffffffffu, src != nullptr);
    const uint32_t bar = bulk::SmemAddr(bars + buf);
    asm volatile("fence.proxy.async;" ::: "memory");
    if (lane == 0) bulk::MbarExpectTx(bar, __popc(live) * bytes);
    __syncwarp();
    if (src != nullptr) bulk::Load(dst + lane * pitch, src, bytes, bar);
  }
  // By all threads; after one expired wait nothing is waited for any more (and *status is raised) before Drain.
  __device__ __forceinline__ void Wait(int buf, int* status) {
    if (ok) {
      const uint32_t bar = bulk::SmemAddr(bars + buf), parity = (phases >> buf) & 1;
      ok = false;
      for (uint32_t it = 0; it < (1u << 18) && !ok; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        ok = done != 0;
      }
      if (!ok) atomicExch(status, 1);
    }
    phases ^= 1u << buf;
  }
  // Before the CTA ends: after an expired wait, copies may still be under way into its memory.
  __device__ __forceinline__ void Drain() const {
    if (!ok) DrainRows(bars, kBuffers, phases);
  }
};

// First phase of a backward level, gate gradients: a thread owns one hidden column and every row_step-th row of each
// level, so the column sums for the bias gradient stay in its registers.  Expressions and order are CellBwd's.
// TG: type of the saved gates, TD: type of dA and ZF.
// The columns of a CTA: with one row group its own output columns [n0, n0 + w) -- then a level's gradients read only what
// this CTA wrote into the mailbox, and no grid barrier stands before them; with several, blocks of 64 dealt out over the
// grid together with strips of rows.
constexpr int kColBlock = 64;
template <int K, typename TG, typename TD>
struct GateGradients {
  static constexpr bool kFast = sizeof(TD) == 2;
  int j, row0, row_step, cols;
  bool owner, local;
  float sums[4], wc[kHeadDzPitch];
  // of the next row, everything but its mailbox row
  int ch[K];
  bool has_parent;
  float gi, go, gu, cown, d_out, gf[K], cch[K];

  __device__ __forceinline__ explicit GateGradients(const NarrowBackwardArgs& a) {
    local = a.row_groups == 1;
    cols = local ? a.w : kColBlock;
    const int col_blocks = (a.H + cols - 1) / cols, strips = local ? 1 : max(1, static_cast<int>(gridDim.x) / col_blocks);
    const int strip = blockIdx.x / col_blocks, lanes = kThreads / cols;
    j = (blockIdx.x % col_blocks) * cols + threadIdx.x % cols;
    row0 = strip * lanes + static_cast<int>(threadIdx.x) / cols;
    row_step = strips * lanes;
    owner = j < a.H && strip < strips;
#pragma unroll
    for (int g = 0; g < 4; ++g) sums[g] = 0.0f;
#pragma unroll
    for (int c = 0; c < kHeadDzPitch; ++c) wc[c] = owner && a.dz != nullptr && c < a.C ? a.Wc[static_cast<size_t>(c) * a.H + j] : 0.0f;
  }
  __device__ __forceinline__ void Fetch(const NarrowBackwardArgs& a, size_t t) {
    const int H = a.H;
    has_parent = __ldg(a.parent + t) >= 0;
    const TG* g = static_cast<const TG*>(a.gates) + t * a.pitch3 + j;
    const TG* f = static_cast<const TG*>(a.gates_f) + t * a.pitch_f + j;
    gi = LoadCg(g); go = LoadCg(g + H); gu = LoadCg(g + 2 * H);
    cown = __ldcg(a.state + t * 2 * H + H + j);
#pragma unroll
    for (int c = 0; c < K; ++c) {
      ch[c] = __ldg(a.child + static_cast<size_t>(c) * a.n_total + t);
      const int chs = a.child_state ? __ldg(a.child_state + static_cast<size_t>(c) * a.n_total + t) : ch[c];
      gf[c] = LoadCg(f + c * H);
      cch[c] = ch[c] >= 0 ? __ldcg(a.state + static_cast<size_t>(chs) * 2 * H + H + j) : 0.0f;
    }
    d_out = 0.0f;
    if (a.dz != nullptr) {
#pragma unroll
      for (int c = 0; c < kHeadDzPitch; ++c)
        if (c < a.C) d_out = fmaf(__ldg(a.dz + t * kHeadDzPitch + c), wc[c], d_out);
    } else {
      d_out = __ldg(a.dOut + t * H + j);
    }
  }
  // Requests the first row of a level whose mailbox rows are not complete yet.
  __device__ __forceinline__ void Request(const NarrowBackwardArgs& a, int off, int end) {
    if (owner && off + row0 < end) Fetch(a, off + row0);
  }
  __device__ __forceinline__ void Level(const NarrowBackwardArgs& a, int off, int end) {
    if (!owner) return;
    const int H = a.H;
    for (int t_ = off + row0; t_ < end; t_ += row_step) {
      const size_t t = t_;
      const float mh = has_parent ? __ldcg(a.mailbox + t * 2 * H + j) : 0.0f, mc = has_parent ? __ldcg(a.mailbox + t * 2 * H + H + j) : 0.0f;
      const GateGradients x = *this;
      if (t_ + row_step < end) Fetch(a, t_ + row_step);   // beside this row's mailbox
      const float dh = x.d_out + mh, th = Tanh<kFast>(x.cown), d_o = dh * th;
      const float dc = mc + (dh * x.go) * (1.0f - th * th);
      const float zi = (dc * x.gu) * x.gi * (1.0f - x.gi), zo = d_o * x.go * (1.0f - x.go), zu = (dc * x.gi) * (1.0f - x.gu * x.gu);
      float zfs = 0.0f;
      TD* zf = static_cast<TD*>(a.ZF) + t * K * H + j;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        float z = 0.0f;
        if (x.ch[c] >= 0) {
          z = (dc * x.cch[c]) * x.gf[c] * (1.0f - x.gf[c]);
          zfs += z;
          a.mailbox[static_cast<size_t>(x.ch[c]) * 2 * H + H + j] = dc * x.gf[c];
        }
        StoreAs(zf + c * H, z);
      }
      TD* d = static_cast<TD*>(a.dA) + t * 4 * H + j;
      StoreAs(d, zi); StoreAs(d + H, zo); StoreAs(d + 2 * H, zu); StoreAs(d + 3 * H, zfs);
      sums[0] += zi; sums[1] += zo; sums[2] += zu; sums[3] += zfs;
    }
  }
  // Column sums of this CTA's rows, row lanes folded in order, into its row of dB_part; scratch: 4 x kThreads floats.
  __device__ __forceinline__ void FoldSums(const NarrowBackwardArgs& a, float* scratch) {
    if (a.dB_part == nullptr) return;
    __syncthreads();
#pragma unroll
    for (int g = 0; g < 4; ++g) scratch[g * kThreads + threadIdx.x] = sums[g];
    __syncthreads();
    if (!owner || threadIdx.x >= cols) return;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float acc = 0.0f;
      for (int r = 0; r < kThreads / cols; ++r) acc += scratch[g * kThreads + r * cols + threadIdx.x];
      a.dB_part[static_cast<size_t>(blockIdx.x) * 4 * a.H + g * a.H + j] += acc;
    }
  }
};

template <auto kKernel, typename Args>
int LaunchCooperative(const Args& args, int grid, size_t smem, cudaStream_t st) {
  static bool configured[kMaxDevices] = {};
  const int dev = CurrentDevice();
  if (!configured[dev]) {
    CAVS_CUDA(cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxSmem)));
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // all CTAs resident, or the launch fails: the barrier needs it
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CAVS_CUDA(cudaLaunchKernelEx(&cfg, kKernel, args));
  CAVS_LAUNCH_CHECK("narrow levels");
  return CAVS_OK;
}
}  // namespace narrow
}  // namespace cavs_b200
#endif
