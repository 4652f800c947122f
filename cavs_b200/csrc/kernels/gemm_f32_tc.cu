// fp32 GEMM on the tensor cores: every fp32 operand value is split into three bf16 values whose sum is the value
// itself (8 + 8 + 8 significant bits), and a product a.b becomes the six bf16 products that carry its leading 24 bits
// (hh | hm, mh, hl, lh, mm; the dropped ones are below 2^-24 of the product).  tcgen05 forms them exactly and sums in
// fp32.
//
// Precision.  The tensor core's additions into an accumulator truncate, so a long chain of them would drift where
// FFMA's rounded additions do not.  Two measures keep the result close to 64 bits: the leading products hh have an
// accumulator of their own that takes only the four MMAs of one 64-wide k block and is then added, rounded, to a register;
// the five correction products, 2^-8 of the size, share a second accumulator that is drained every 512 k.
//   |err| / |C| against 64 bits (2-norm), FFMA kernel -> this one:
//   normal values         k = 16: 7.4e-8 -> 3.6e-8;  150: 2.2e-7 -> 7.6e-8;  512: 4.1e-7 -> 9.0e-8;  14474: 2.2e-6 -> 3.0e-7
//   uniform in 0..1       k = 16: 6.2e-8 -> 3.8e-8;   64: 1.2e-7 -> 8.2e-8;  512: 3.1e-7 -> 8.6e-8;  14474: 1.7e-6 -> 2.4e-7
//   half-normal           k = 16: 6.2e-8 -> 3.9e-8;   64: 1.2e-7 -> 8.9e-8;  512: 3.5e-7 -> 9.6e-8;  14474: 1.8e-6 -> 2.6e-7
//   sigmoids of normal    k = 16: 6.1e-8 -> 2.7e-8;   64: 1.1e-7 -> 4.1e-8;  512: 3.0e-7 -> 5.6e-8;  14474: 1.7e-6 -> 2.3e-7
// (of one sign, the truncation is a bias of -1.5e-8 to -8e-8).  Further off than the FFMA kernel where few terms of one sign
// make up a sum over a short k -- exp(2 x normal): k = 8: 4.2e-8 -> 1.0e-7; 64: 1.9e-7 -> 4.9e-7; closer again from 512 on --
// where all values lie within 1 % of 2 at k = 14474 (1.7e-6 -> 1.8e-6), and where results lie below 2^-120, whose corrections
// reach fp32's subnormals (2^-124: 4.0e-7 -> 4.6e-7).
//
// What bounds it: 127 TFLOP/s of fp32 products at [14474, 512] x [512, 10000] (5846 us with the FFMA kernel, 1163 with
// this one), 110 with k = 10000 (6858, 1352), 93 with k = 14474 and both operands strided along k (6989, 1598).  Of these
// 0, 1 and 9 % are the price of looking at every split for bits that its three parts do not hold.  Six MMAs per product stand
// against operands that must be split by ordinary instructions.  Per 128 x 128 x 64
// block the MMAs take 1536 clocks of the tensor pipe, the split of 2 x 8192 values ~1000 issue slots of each scheduler; the block takes 4200,
// because the splitting warps wait for their loads (long-scoreboard stalls, tensor pipe 35 % busy).  Tried against that:
// reloading run by run, a second set of registers under setmaxnreg, clamped instead of predicated addresses -- all slower.
// So the split is done in the kernel (no extra pass over memory, no copies of the weights to keep) by eight warps that
// load the next block's values while they convert this one's, beside eight warps that issue the MMAs and drain the
// accumulators.
//
//   warps 0..7   accumulators: TMEM -> registers every k block, the tile's store; one lane of warp 0 issues the
//                MMAs, one block ahead of the drain (a seventeenth warp would cut every thread to 96 registers)
//   warps 8..15  operands: global -> registers -> three bf16 planes in 128-byte-swizzled shared memory
//
// A value that its three parts do not hold -- infinity, NaN, beyond bf16's largest, or below 2^-110 with bits that reach under
// bf16's smallest subnormal, 2^-133 -- marks its tile, which is computed by plain fp32 loops after all others: such operands give
// what fp32 arithmetic gives.  So does a tile whose bounded waits expire, row by row.
#include <cuda_bf16.h>

#include <cstdint>

#include "abi_common.h"
#include "kernels/gemm.h"
#include "kernels/gemm_tc.cuh"
#include "kernels/launch.h"

namespace cavs_b200 {
namespace {

using namespace tc;   // mbarrier, TMEM and MMA wrappers of the bf16 GEMM

constexpr int kDrainWarps = 8, kSplitWarps = 8;
constexpr int kF32Threads = (kDrainWarps + kSplitWarps) * 32;
constexpr int kSplitThreads = kSplitWarps * 32;
constexpr int kMarks = 4096;     // tiles per CTA that can be marked one by one (the last bit stands for all from there on)
constexpr int kCorrBlocks = 8;   // k blocks per drain of the correction accumulator

template <int kBN>
struct SplitSmem {
  static constexpr int kAPlane = kBM * 128, kBPlane = kBN * 128;   // 64 bf16 per row
  static constexpr int kStage = 3 * (kAPlane + kBPlane);
  static constexpr int kStages = 2;
  static constexpr int kCOff = kStages * kStage;
  static constexpr int kBarOff = kCOff + kDrainWarps * 32 * 128;
  static constexpr int kBytes = kBarOff + 96 + kMarks / 8 + 1024;   // barriers, TMEM address, marks; alignment
};

struct SplitParams {
  GemmF32Args g;
  int n_splits, kb_per_split;
  long long split_stride;
  int chain_early;
  int withhold;   // wait self-test: no operand is ever ready
};

// Bounded wait (about 0.3 s) whose polls suspend the warp in hardware, so that waiting warps leave the issue slots to
// the warps that split.
__device__ __forceinline__ bool WaitPhase(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < (1u << 18); ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// The same by a whole warp, with one outcome for all lanes: warp-wide instructions follow.  (The vote stands inside the poll:
// a vote on the outcome cost 100 bytes of spilled registers.)
__device__ __forceinline__ bool WaitPhaseWarp(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < (1u << 18); ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "vote.sync.all.pred q, p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Position of one k block in this CTA's list of (tile, k split) work items.
struct BlockPos {
  int w, i, kb_count, m0, n0, k0, t_local;
};

template <int kBN>
__device__ __forceinline__ bool SeekItem(const SplitParams& p, int n_work, int tiles_n, BlockPos& b) {
  if (b.w >= n_work) return false;
  const int z = b.w % p.n_splits, tile = b.w / p.n_splits;
  const int kb_begin = z * p.kb_per_split;
  b.kb_count = min(p.kb_per_split, (p.g.k + kBK - 1) / kBK - kb_begin);
  b.m0 = (tile / tiles_n) * kBM;
  b.n0 = (tile % tiles_n) * kBN;
  b.k0 = kb_begin * kBK;
  b.i = 0;
  return true;
}

__device__ __forceinline__ uint32_t Bits(__nv_bfloat162 x) { return *reinterpret_cast<uint32_t*>(&x); }

// Splits eight values and stores them as one 16-byte word of each plane.  `rest` collects the bits of what the third part
// has to hold: those below bf16's sixteen are set when it cannot (a value without a finite split leaves NaN there, infinity -
// infinity).  One three-input OR per pair of values.
__device__ __forceinline__ void StoreSplit(const float (&v)[8], uint32_t dst, int plane_bytes, uint32_t& rest) {
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float x = v[2 * e], y = v[2 * e + 1];
    const __nv_bfloat162 hi = __floats2bfloat162_rn(x, y);
    x -= __low2float(hi); y -= __high2float(hi);
    const __nv_bfloat162 mid = __floats2bfloat162_rn(x, y);
    x -= __low2float(mid); y -= __high2float(mid);
    rest |= __float_as_uint(x) | __float_as_uint(y);
    const __nv_bfloat162 lo = __floats2bfloat162_rn(x, y);
    h[e] = Bits(hi); m[e] = Bits(mid); l[e] = Bits(lo);
  }
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + plane_bytes), "r"(m[0]), "r"(m[1]), "r"(m[2]), "r"(m[3]) : "memory");
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 2 * plane_bytes), "r"(l[0]), "r"(l[1]), "r"(l[2]), "r"(l[3]) : "memory");
}

// How an operand is read: k contiguous, or rows contiguous, in aligned 16-byte words; k contiguous; any other strides.
enum ReadMode : int { kStrided = 0, kRunsOfK = 1, kRunsOfK16 = 2, kRows16 = 3 };

// A value inside [0, valid), zero outside, without a branch: the compiler keeps a block's loads in flight across the
// conversion of the previous block (behind a branch it waits for them where the paths meet).
__device__ __forceinline__ void LoadIf(bool pred, const float* src, float& v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@p ld.global.nc.f32 %0, [%1];\n\t}"
               : "=&f"(v) : "l"(src), "r"(static_cast<int>(pred)));
}
__device__ __forceinline__ void LoadIf4(bool pred, const float* src, float& a, float& b, float& c, float& d) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
      "@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=&f"(a), "=&f"(b), "=&f"(c), "=&f"(d)
      : "l"(src), "r"(static_cast<int>(pred)));
}

// One operand's tile of a k block: each thread holds kChunks runs of eight k values.  rs: stride between rows, cs:
// between k values.  Rows and k values past the end are zeros.
template <int kRows, int kMode>
struct OperandTile {
  static constexpr int kChunks = kRows * 8 / kSplitThreads;
  float v[kChunks][8];
  // Row and k run of chunk c.  Neighbouring lanes read neighbouring addresses, and any eight of them store to
  // eight different 16-byte columns of the swizzled rows (no bank conflicts).
  static __device__ __forceinline__ void Pos(int tid, int c, int& r, int& j) {
    const int idx = tid + c * kSplitThreads;
    if (kMode == kStrided) { r = idx & (kRows - 1); j = idx / kRows; }
    else if (kMode == kRows16) { r = ((tid >> 2) & 7) * 4 + (tid >> 6) * 32 + c; j = (tid & 3) + ((tid >> 5) & 1) * 4; }
    else { r = idx >> 3; j = idx & 7; }
  }
  __device__ __forceinline__ void Load(const float* base, long long rs, long long cs, int row0, int rows, int k0, int k_end, int tid) {
    if constexpr (kMode == kRows16) {
      static_assert(kMode != kRows16 || kChunks == 4, "four rows per 16-byte load");
      int r, j;
      Pos(tid, 0, r, j);
      const int k = k0 + j * 8, valid = row0 + r < rows ? k_end - k : 0;
      const float* src = base + row0 + r + k * cs;
#pragma unroll
      for (int e = 0; e < 8; ++e) LoadIf4(valid > e, src + e * cs, v[0][e], v[1][e], v[2][e], v[3][e]);
    } else {
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        int r, j;
        Pos(tid, c, r, j);
        const int row = row0 + r, k = k0 + j * 8, valid = row < rows ? k_end - k : 0;
        const float* src = base + row * rs + (kMode == kStrided ? k * cs : k);
        if constexpr (kMode == kRunsOfK16) {
          LoadIf4(valid > 0, src, v[c][0], v[c][1], v[c][2], v[c][3]);
          LoadIf4(valid > 4, src + 4, v[c][4], v[c][5], v[c][6], v[c][7]);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) LoadIf(valid > e, src + (kMode == kStrided ? e * cs : e), v[c][e]);
        }
      }
    }
  }
  __device__ __forceinline__ void Store(uint32_t dst, int tid, uint32_t& rest) const {
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      int r, j;
      Pos(tid, c, r, j);
      StoreSplit(v[c], dst + r * 128 + ((j ^ (r & 7)) << 4), kRows * 128, rest);
    }
  }
};

// acc += accumulator columns, 16 at a time (beside the accumulators' 64 registers)
template <int kCols>
__device__ __forceinline__ void DrainAdd(float (&acc)[kCols], uint32_t taddr) {
#pragma unroll
  for (int c0 = 0; c0 < kCols; c0 += 16) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr + c0));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(r[j]);
  }
}

// One row of a tile's columns [col0, col0 + cols) in fp32, by one thread that waits for nobody: after an expired wait.
__device__ __noinline__ void PlainRow(const float* a, long long a_rs, long long a_cs, const float* b, long long b_rs, long long b_cs, int m, int n, float* c, long long ldc, int accumulate, int row, int col0, int cols, int k0,
                                      int k1) {
  if (row >= m) return;
  for (int j = col0; j < min(col0 + cols, n); ++j) {
    float acc = 0.0f;
    for (int k = k0; k < k1; ++k) acc = fmaf(a[row * a_rs + k * a_cs], b[k * b_rs + j * b_cs], acc);
    float* dst = c + row * ldc + j;
    *dst = accumulate ? *dst + acc : acc;
  }
}

// A whole tile in fp32 by all threads, k ascending: 8 x kBN / 32 outputs per thread in a 16 x 32 grid of threads, 32 k values
// staged at a time in the operands' shared memory, the next ones in flight meanwhile.
template <int kBN>
__device__ __forceinline__ void PlainTile(const GemmF32Args& g, float* c, long long ldc, int accumulate, int m0, int n0, int k0, int k1,
                                       float* stage) {
  constexpr int kC = kBN / 32, kStep = 32, kPitchA = kBM + 4, kPitchB = kBN + 4;
  constexpr int kLoadA = kBM * kStep / kF32Threads, kLoadB = kBN * kStep / kF32Threads;
  float *as = stage, *bs = stage + kStep * kPitchA;
  const int tc = threadIdx.x & 31, tr = threadIdx.x >> 5;
  float acc[8][kC], va[kLoadA], vb[kLoadB];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < kC; ++j) acc[i][j] = 0.0f;
  // element e of a thread: neighbouring threads read along the operand's contiguous direction
  const bool a_k = g.a_cs == 1, b_k = g.b_rs == 1;
  auto at_a = [&](int e, int& r, int& k) { const int i = threadIdx.x + e * kF32Threads; if (a_k) { k = i % kStep; r = i / kStep; } else { r = i % kBM; k = i / kBM; } };
  auto at_b = [&](int e, int& j, int& k) { const int i = threadIdx.x + e * kF32Threads; if (b_k) { k = i % kStep; j = i / kStep; } else { j = i % kBN; k = i / kBN; } };
  auto load = [&](int kb) {
    int r, k;
#pragma unroll
    for (int e = 0; e < kLoadA; ++e) { at_a(e, r, k); va[e] = m0 + r < g.m && kb + k < k1 ? g.a[(m0 + r) * g.a_rs + (kb + k) * g.a_cs] : 0.0f; }
#pragma unroll
    for (int e = 0; e < kLoadB; ++e) { at_b(e, r, k); vb[e] = n0 + r < g.n && kb + k < k1 ? g.b[(kb + k) * g.b_rs + (n0 + r) * g.b_cs] : 0.0f; }
  };
  load(k0);
  for (int kb = k0; kb < k1; kb += kStep) {
    int r, k;
    __syncthreads();   // the previous values' readers are done
#pragma unroll
    for (int e = 0; e < kLoadA; ++e) { at_a(e, r, k); as[k * kPitchA + r] = va[e]; }
#pragma unroll
    for (int e = 0; e < kLoadB; ++e) { at_b(e, r, k); bs[k * kPitchB + r] = vb[e]; }
    __syncthreads();
    load(kb + kStep);
#pragma unroll 8
    for (int u = 0; u < kStep; ++u) {
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        const float4 t = *reinterpret_cast<const float4*>(as + u * kPitchA + tr * 8 + i);
        x[i] = t.x; x[i + 1] = t.y; x[i + 2] = t.z; x[i + 3] = t.w;
      }
#pragma unroll
      for (int j = 0; j < kC; ++j) {
        const float y = bs[u * kPitchB + j * 32 + tc];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(x[i], y, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < kC; ++j) {
      const int row = m0 + tr * 8 + i, col = n0 + j * 32 + tc;
      if (row >= g.m || col >= g.n) continue;
      float* dst = c + row * ldc + col;
      *dst = accumulate ? *dst + acc[i][j] : acc[i][j];
    }
}

// The marked tiles of this CTA, after all others: nobody waits for them then, and a function of its own, called where nothing
// else is live, leaves the registers of the loops alone.  [14474, 512] x [512, 10000] with every tile marked: 7.3 ms (FFMA
// kernel 5.7; one thread per row 45 or more), with one marked 1.29 (1.15 without).
template <int kBN>
__device__ __noinline__ void PlainTiles(const SplitParams& p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t* marks = reinterpret_cast<const uint32_t*>(smem + SplitSmem<kBN>::kBarOff) + 24;
  const int tiles_n = (p.g.n + kBN - 1) / kBN, n_work = ((p.g.m + kBM - 1) / kBM) * tiles_n * p.n_splits;
  for (int i = 0; i < kMarks / 32; ++i)
    for (uint32_t word = marks[i]; word != 0; word &= word - 1) {
      BlockPos b;
      b.w = blockIdx.x + (i * 32 + __ffs(word) - 1) * gridDim.x;
      if (i * 32 + __ffs(word) == kMarks || !SeekItem<kBN>(p, n_work, tiles_n, b)) continue;
      const bool part = p.n_splits > 1;
      PlainTile<kBN>(p.g, part ? p.g.scratch + (b.w % p.n_splits) * p.split_stride : p.g.c, part ? p.g.n : p.g.ldc, part ? 0 : p.g.accumulate, b.m0,
                     b.n0, b.k0, min(p.g.k, b.k0 + b.kb_count * kBK), reinterpret_cast<float*>(smem));
    }
}

// (A parameter whose address is taken is copied to the stack at entry unless it is a grid constant: with the marks asked before
// PlainTiles is called, [256, 512] x [512, 1536] went from 20.4 to 18.5 us, [595, 150] x [150, 450] from 18.4 to 16.4.)
template <int kBN, int kModeA, int kModeB>
__global__ void __launch_bounds__(kF32Threads, 1) GemmF32SplitKernel(const __grid_constant__ SplitParams p) {
  using S = SplitSmem<kBN>;
  constexpr int kCols = kBN / 2;   // columns per drain warp
  ChainRelease(p.chain_early);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBarOff);
  uint64_t *full = bars, *empty = bars + 2, *main_full = bars + 4, *main_empty = bars + 6, *corr_empty = bars + 8, *drained = bars + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  uint32_t* any_mark = tmem_slot + 1;
  uint32_t* marks = reinterpret_cast<uint32_t*>(bars + 12);   // one bit per tile of this CTA with operands that have no exact split

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const GemmF32Args& g = p.g;
  const int tiles_n = (g.n + kBN - 1) / kBN;
  const int n_work = ((g.m + kBM - 1) / kBM) * tiles_n * p.n_splits;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      MbarInit(SmemAddr(full + s), kSplitWarps);
      MbarInit(SmemAddr(empty + s), 1);
      MbarInit(SmemAddr(main_full + s), 1);
      MbarInit(SmemAddr(main_empty + s), kDrainWarps);
      MbarInit(SmemAddr(corr_empty + s), kDrainWarps);
    }
    MbarInit(SmemAddr(drained), 1);
    *any_mark = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < kMarks / 32; i += kF32Threads) marks[i] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(tmem_slot)), "r"(4 * kBN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  bool ok = true;
  ChainAcquire();

  if (warp >= kDrainWarps) {
    // ---- operands ----
    const int tid = threadIdx.x - kDrainWarps * 32;
    OperandTile<kBM, kModeA> ta;
    OperandTile<kBN, kModeB> tb;
    BlockPos nxt;   // the next block to load
    nxt.w = blockIdx.x; nxt.t_local = 0;
    bool have = SeekItem<kBN>(p, n_work, tiles_n, nxt) && !p.withhold;   // (the grid is no larger than the work list)
    ta.Load(g.a, g.a_rs, g.a_cs, nxt.m0, g.m, nxt.k0, g.k, tid);
    tb.Load(g.b, g.b_cs, g.b_rs, nxt.n0, g.n, nxt.k0, g.k, tid);
    for (uint32_t it = 0; have; ++it) {
      const int t_local = nxt.t_local;
      if (++nxt.i < nxt.kb_count) {
        nxt.k0 += kBK;
      } else {
        nxt.w += gridDim.x;
        ++nxt.t_local;
        have = SeekItem<kBN>(p, n_work, tiles_n, nxt);
        if (!have) nxt.k0 = g.k;   // nothing follows: loads of zeros, so that the loads stand behind no branch
      }
      const int s = it & 1;
      ok = WaitPhaseWarp(SmemAddr(empty + s), ((it >> 1) & 1) ^ 1);
      if (!ok) break;
      const uint32_t a_dst = SmemAddr(smem + s * S::kStage), b_dst = a_dst + 3 * S::kAPlane;
      uint32_t rest_a = 0, rest_b = 0;
      ta.Store(a_dst, tid, rest_a);
      ta.Load(g.a, g.a_rs, g.a_cs, nxt.m0, g.m, nxt.k0, g.k, tid);
      tb.Store(b_dst, tid, rest_b);
      tb.Load(g.b, g.b_cs, g.b_rs, nxt.n0, g.n, nxt.k0, g.k, tid);
      if (((rest_a | rest_b) & 0xffffu) != 0) {
        atomicOr(marks + (min(t_local, kMarks - 1) >> 5), 1u << (min(t_local, kMarks - 1) & 31));
        *any_mark = 1;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) MbarArrive(SmemAddr(full + s));
    }
  } else {
    // ---- MMAs ----
    BlockPos mma;
    mma.w = blockIdx.x; mma.t_local = 0;
    uint32_t mma_it = 0, mma_ci = 0;
    bool mma_more = SeekItem<kBN>(p, n_work, tiles_n, mma);
    auto issue = [&]() {   // one k block, by one lane of warp 0
      constexpr uint32_t idesc = InstrDesc(kMajorK, kMajorK, kBN, kBM);
      constexpr uint32_t step = kUmmaK * 2 >> 4;
      const int s = mma_it & 1;
      const bool corr_first = mma.i % kCorrBlocks == 0;
      if (!WaitPhase(SmemAddr(full + s), (mma_it >> 1) & 1)) return false;
      if (!WaitPhase(SmemAddr(main_empty + s), ((mma_it >> 1) & 1) ^ 1)) return false;
      if (corr_first && !WaitPhase(SmemAddr(corr_empty + (mma_ci & 1)), ((mma_ci >> 1) & 1) ^ 1)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a_addr = SmemAddr(smem + s * S::kStage);
      const uint64_t a = SmemDesc(a_addr, kMajorK), b = SmemDesc(a_addr + 3 * S::kAPlane, kMajorK);
      constexpr uint32_t pa = S::kAPlane >> 4, pb = S::kBPlane >> 4;
      const uint32_t d_main = tmem + s * kBN, d_corr = tmem + (2 + (mma_ci & 1)) * kBN;
#pragma unroll
      for (int kk = 0; kk < kBK / kUmmaK; ++kk) {
        const uint64_t ak = a + kk * step, bk = b + kk * step;
        UmmaBf16(d_main, ak, bk, idesc, kk > 0 ? 1u : 0u);
        UmmaBf16(d_corr, ak + 2 * pa, bk, idesc, (!corr_first || kk > 0) ? 1u : 0u);   // smallest first: l.h, h.l, m.m, m.h, h.m
        UmmaBf16(d_corr, ak, bk + 2 * pb, idesc, 1u);
        UmmaBf16(d_corr, ak + pa, bk + pb, idesc, 1u);
        UmmaBf16(d_corr, ak + pa, bk, idesc, 1u);
        UmmaBf16(d_corr, ak, bk + pb, idesc, 1u);
      }
      UmmaCommit(SmemAddr(empty + s));
      UmmaCommit(SmemAddr(main_full + s));
      return true;
    };
    auto issue_next = [&]() {   // all of warp 0
      if (!mma_more || !ok) return;
      bool good = true;
      if (lane == 0) good = issue();
      ok = __all_sync(0xffffffffu, good);
      ++mma_it;
      if (mma.i % kCorrBlocks == kCorrBlocks - 1 || mma.i == mma.kb_count - 1) ++mma_ci;
      if (++mma.i == mma.kb_count) {
        mma.w += gridDim.x;
        mma_more = SeekItem<kBN>(p, n_work, tiles_n, mma);
      }
    };
    if (warp == 0) issue_next();
    // ---- accumulators and stores ----
    const int quarter = warp & 3, half = warp >> 2;
    uint32_t it = 0, ci = 0;
    BlockPos b;
    b.t_local = 0;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + half * kCols;
    const uint32_t slot = SmemAddr(smem + S::kCOff) + warp * 32 * 128;
    for (b.w = blockIdx.x; SeekItem<kBN>(p, n_work, tiles_n, b); b.w += gridDim.x, ++b.t_local) {
      float acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0.0f;
      for (int i = 0; i < b.kb_count && ok; ++i, ++it) {
        const int s = it & 1;
        if (warp == 0) issue_next();   // the block after this one: its MMAs follow this block's without a gap
        ok = ok && WaitPhaseWarp(SmemAddr(main_full + s), (it >> 1) & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const bool corr_last = i % kCorrBlocks == kCorrBlocks - 1 || i == b.kb_count - 1;
        DrainAdd<kCols>(acc, lane_addr + s * kBN);
        if (corr_last) DrainAdd<kCols>(acc, lane_addr + (2 + (ci & 1)) * kBN);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          MbarArrive(SmemAddr(main_empty + s));
          if (corr_last) MbarArrive(SmemAddr(corr_empty + (ci & 1)));
        }
        if (corr_last) ++ci;
      }
      const int z = b.w % p.n_splits;
      float* c = p.n_splits > 1 ? g.scratch + z * p.split_stride : g.c;
      const long long ldc = p.n_splits > 1 ? g.n : g.ldc;
      const int accumulate = p.n_splits > 1 ? 0 : g.accumulate;
      const int row0 = b.m0 + quarter * 32, col_base = b.n0 + half * kCols;
      const int mark = min(b.t_local, kMarks - 1);
      const bool marked = *reinterpret_cast<volatile uint32_t*>(marks + (mark >> 5)) >> (mark & 31) & 1;
      if (!ok || marked) {   // marked: computed after all others, but for the tiles that share the last bit
        if (!marked || mark == kMarks - 1) PlainRow(g.a, g.a_rs, g.a_cs, g.b, g.b_rs, g.b_cs, g.m, g.n, c, ldc, accumulate, row0 + lane, col_base, kCols, b.k0, min(g.k, b.k0 + b.kb_count * kBK));
        continue;
      }
      const bool vec = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0;
#pragma unroll
      for (int c0 = 0; c0 < kCols; c0 += 32) {
        const int col0 = col_base + c0;
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(slot + lane * 128 + ((q ^ (lane & 7)) << 4)),
                       "r"(__float_as_uint(acc[c0 + 4 * q])), "r"(__float_as_uint(acc[c0 + 4 * q + 1])),
                       "r"(__float_as_uint(acc[c0 + 4 * q + 2])), "r"(__float_as_uint(acc[c0 + 4 * q + 3])) : "memory");
        __syncwarp();
        if (vec && col0 + 32 <= g.n) {
          // eight lanes per row, four rows per instruction: full 128-byte lines
          const int q = lane & 7;
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const int i = t * 4 + (lane >> 3);
            if (row0 + i >= g.m) continue;
            float4 v;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(slot + i * 128 + ((q ^ (i & 7)) << 4)) : "memory");
            float4* dst = reinterpret_cast<float4*>(c + (row0 + i) * ldc + col0 + 4 * q);
            if (accumulate) {
              const float4 o = *dst;
              v.x = o.x + v.x; v.y = o.y + v.y; v.z = o.z + v.z; v.w = o.w + v.w;
            }
            *dst = v;
          }
        } else if (col0 + lane < g.n) {
          for (int i = 0; i < min(32, g.m - row0); ++i) {
            float v;
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(slot + i * 128 + (((lane >> 2) ^ (i & 7)) << 4) + (lane & 3) * 4) : "memory");
            float* dst = c + (row0 + i) * ldc + col0 + lane;
            *dst = accumulate ? *dst + v : v;
          }
        }
      }
    }
    if (warp == 0 && !ok) {   // the accumulators are given back when no MMA is under way any more
      if (lane == 0) {
        UmmaCommit(SmemAddr(drained));
        WaitPhase(SmemAddr(drained), 0);
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(4 * kBN));
  // (asked before the call, which would save registers first; the address is formed anew, not kept)
  uint32_t any;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(any) : "r"(((SmemAddr(smem_raw) + 1023) & ~1023u) + S::kBarOff + 23 * 4) : "memory");
  if (any != 0) PlainTiles<kBN>(p);
}

ReadMode ReadModeOf(const float* base, int rows, long long row_stride, int k, long long k_stride, int tile_rows) {
  const bool aligned = reinterpret_cast<uintptr_t>(base) % 16 == 0;
  if (k_stride == 1) return aligned && row_stride % 4 == 0 && k % 4 == 0 ? kRunsOfK16 : kRunsOfK;
  return aligned && row_stride == 1 && k_stride % 4 == 0 && rows % 4 == 0 && tile_rows == 128 ? kRows16 : kStrided;
}

template <int kBN, int kModeA, int kModeB>
int LaunchSplit(const SplitParams& p, cudaStream_t stream) {
  constexpr int bytes = SplitSmem<kBN>::kBytes;
  static bool configured[kMaxDevices] = {};
  const int dev = CurrentDevice();
  if (!configured[dev]) {
    CAVS_CUDA(cudaFuncSetAttribute(GemmF32SplitKernel<kBN, kModeA, kModeB>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    configured[dev] = true;
  }
  const long long work = static_cast<long long>((p.g.m + kBM - 1) / kBM) * ((p.g.n + kBN - 1) / kBN) * p.n_splits;
  const int grid = static_cast<int>(std::min<long long>(work, SmCount()));
  CAVS_CUDA(LaunchChained(GemmF32SplitKernel<kBN, kModeA, kModeB>, dim3(grid), dim3(kF32Threads), bytes, stream, p));
  CAVS_LAUNCH_CHECK("gemm_f32 split");
  return CAVS_OK;
}
template <int kBN, int kModeA>
int LaunchSplitB(const SplitParams& p, ReadMode b, cudaStream_t stream) {
  switch (b) {
    case kRows16: return LaunchSplit<kBN, kModeA, kBN == 128 ? kRows16 : kStrided>(p, stream);
    case kRunsOfK16: return LaunchSplit<kBN, kModeA, kRunsOfK16>(p, stream);
    case kRunsOfK: return LaunchSplit<kBN, kModeA, kRunsOfK>(p, stream);
    default: return LaunchSplit<kBN, kModeA, kStrided>(p, stream);
  }
}
template <int kBN>
int LaunchSplitAB(const SplitParams& p, ReadMode a, ReadMode b, cudaStream_t stream) {
  switch (a) {
    case kRows16: return LaunchSplitB<kBN, kRows16>(p, b, stream);
    case kRunsOfK16: return LaunchSplitB<kBN, kRunsOfK16>(p, b, stream);
    case kRunsOfK: return LaunchSplitB<kBN, kRunsOfK>(p, b, stream);
    default: return LaunchSplitB<kBN, kStrided>(p, b, stream);
  }
}

}  // namespace

int GemmF32Split(const GemmF32Args& g, int tile_n, int* splits, cudaStream_t stream) {
  SplitParams p;
  p.g = g;
  const int kb = (g.k + kBK - 1) / kBK;
  p.kb_per_split = (kb + *splits - 1) / *splits;
  p.n_splits = *splits = (kb + p.kb_per_split - 1) / p.kb_per_split;
  p.split_stride = static_cast<long long>(g.m) * g.n;
  p.chain_early = ChainEarly();
  p.withhold = g.withhold;
  const ReadMode ma = ReadModeOf(g.a, g.m, g.a_rs, g.k, g.a_cs, kBM), mb = ReadModeOf(g.b, g.n, g.b_cs, g.k, g.b_rs, tile_n);
  return tile_n == 128 ? LaunchSplitAB<128>(p, ma, mb, stream) : LaunchSplitAB<64>(p, ma, mb, stream);
}

}  // namespace cavs_b200
