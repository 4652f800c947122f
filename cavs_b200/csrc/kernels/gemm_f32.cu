// fp32 GEMM, used by the fp32 configurations whose results must stay within 1e-5 relative of the reference's
// cublasSgemm calls (cavs/backend/cublas_wrapper.cc:13-28): the choice between the tensor-core kernel on split operands
// (gemm_f32_tc.cu) and, for products too small for it, the CUDA cores (FFMA) -- a 64x64x16 register-tiled kernel with
// element strides (any transpose without a copy) and a software-pipelined k loop whose sum over k runs in ascending
// order within a thread.
#include <cstdint>

#include "abi_common.h"
#include "kernels/gemm.h"
#include "kernels/launch.h"

#include <algorithm>

namespace cavs_b200 {
namespace {

constexpr int kTM = 64, kTN = 64, kTK = 16;

// One k-step's share of the A and B tiles for this thread: 4 elements each (tiles are 64 x 16 and 16 x 64).
struct TileRegs { float a[4], b[4]; };

__device__ __forceinline__ void LoadTile(const GemmF32Args& g, int m0, int n0, int k0, TileRegs& r) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int idx = threadIdx.x + e * 256;
    // Walk the fastest-varying global dimension with consecutive threads.
    int ai, ak;
    if (g.a_cs == 1) { ak = idx & 15; ai = idx >> 4; } else { ai = idx & 63; ak = idx >> 6; }
    const int gi = m0 + ai, gk = k0 + ak;
    r.a[e] = (gi < g.m && gk < g.k) ? g.a[gi * g.a_rs + gk * g.a_cs] : 0.0f;
    int bk, bj;
    if (g.b_cs == 1) { bj = idx & 63; bk = idx >> 6; } else { bk = idx & 15; bj = idx >> 4; }
    const int gj = n0 + bj, gk2 = k0 + bk;
    r.b[e] = (gj < g.n && gk2 < g.k) ? g.b[gk2 * g.b_rs + gj * g.b_cs] : 0.0f;
  }
}
__device__ __forceinline__ void StoreTile(const GemmF32Args& g, float (*sa)[kTM + 4], float (*sb)[kTN + 4], const TileRegs& r) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int idx = threadIdx.x + e * 256;
    int ai, ak;
    if (g.a_cs == 1) { ak = idx & 15; ai = idx >> 4; } else { ai = idx & 63; ak = idx >> 6; }
    sa[ak][ai] = r.a[e];
    int bk, bj;
    if (g.b_cs == 1) { bj = idx & 63; bk = idx >> 6; } else { bk = idx & 15; bj = idx >> 4; }
    sb[bk][bj] = r.b[e];
  }
}

// The k loop is software-pipelined: the next step's operands travel from global memory to registers while the
// current step's tiles (in shared memory, double-buffered) are multiplied, so a step costs its arithmetic and one
// barrier instead of a global-memory round trip -- these GEMMs have few tiles and long k loops (a level of a few
// hundred rows against [H, 4H] weights), i.e. their duration is the k loop's latency.
__global__ void __launch_bounds__(256) GemmF32Kernel(GemmF32Args g) {
  __shared__ float sa[2][kTK][kTM + 4];
  __shared__ float sb[2][kTK][kTN + 4];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * kTM, n0 = blockIdx.x * kTN;
  // k split: CTA z multiplies the k range [z * k_per_split, ...) and stores its partial product into slab z of the scratch
  const int k_begin = g.k_per_split > 0 ? blockIdx.z * g.k_per_split : 0;
  const int k_end = g.k_per_split > 0 ? min(g.k, k_begin + g.k_per_split) : g.k;
  if (g.k_per_split > 0) { g.c = g.scratch + static_cast<size_t>(blockIdx.z) * g.m * g.n; g.ldc = g.n; g.accumulate = 0; }
  g.k = k_end;   // the tile loaders guard against k
  float acc[4][4] = {};
  TileRegs regs;
  LoadTile(g, m0, n0, k_begin, regs);
  StoreTile(g, sa[0], sb[0], regs);
  __syncthreads();
  int cur = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += kTK) {
    const bool more = k0 + kTK < k_end;
    if (more) LoadTile(g, m0, n0, k0 + kTK, regs);
#pragma unroll
    for (int kk = 0; kk < kTK; ++kk) {
      float av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = sa[cur][kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = sb[cur][kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (more) StoreTile(g, sa[cur ^ 1], sb[cur ^ 1], regs);   // the other buffer: last read before the previous barrier
    __syncthreads();
    cur ^= 1;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gi = m0 + ty * 4 + i;
    if (gi >= g.m) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gj = n0 + tx * 4 + j;
      if (gj >= g.n) continue;
      float* dst = g.c + gi * g.ldc + gj;
      *dst = g.accumulate ? *dst + acc[i][j] : acc[i][j];
    }
  }
}

// C[i,j] (+)= sum over splits, in split order
__global__ void __launch_bounds__(256) GemmF32Reduce(float* __restrict__ c, long long ldc, const float* __restrict__ part, int m, int n,
                                                     int splits, int accumulate) {
  ChainAcquire();
  const long long total = static_cast<long long>(m) * n;
  for (long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * 256) {
    float acc = 0.0f;
    for (int z = 0; z < splits; ++z) acc += part[z * total + i];
    float* dst = c + (i / n) * ldc + (i % n);
    *dst = accumulate ? *dst + acc : acc;
  }
}

// k splits of the FFMA kernel: few tiles and a long k loop go to enough CTAs to fill the machine once (at least 64 k
// per split).
int PlainSplits(const GemmF32Args& g, long long tiles, int sms) {
  if (g.scratch_bytes == 0 || tiles >= sms || g.k < 256) return 1;
  int splits = static_cast<int>(std::min<long long>(std::min<long long>(16, g.k / 64), (2LL * sms) / tiles));
  while (splits > 1 && static_cast<size_t>(splits) * g.m * g.n * sizeof(float) > g.scratch_bytes) --splits;
  return splits;
}

// Estimated microseconds, fitted to measurements of both kernels (B200, shapes from [20, 600] x 200 to [14474, 10000] x
// 512, within 15 %).  Second pass over the partial products of a k split: launch + slabs in, result out.
double ReduceCost(const GemmF32Args& g, int splits) {
  return splits > 1 ? 2.0 + 4.0 * (splits + 1) * g.m * g.n / 3e6 : 0.0;
}
// FFMA: a 16-wide k step costs 0.92 us of latency, or 0.77 us of arithmetic for each CTA that shares the SM.
double PlainCost(const GemmF32Args& g, long long tiles, int splits, int sms) {
  const double steps = ((g.k + splits - 1) / splits + kTK - 1) / kTK;
  return 3.5 + steps * std::max(0.92, 0.77 * ((tiles * splits + sms - 1) / sms)) + ReduceCost(g, splits);
}
// Tensor cores: a 64-wide k block costs 2.2 us with 128 columns per tile, 1.95 us with 64.
double SplitCost(const GemmF32Args& g, int tile_n, int splits, int sms) {
  const long long items = static_cast<long long>((g.m + 127) / 128) * ((g.n + tile_n - 1) / tile_n) * splits;
  const long long blocks = ((g.k + 63) / 64 + splits - 1) / splits, waves = (items + sms - 1) / sms;
  return 4.5 + waves * (0.8 + blocks * (tile_n == 128 ? 2.2 : 1.95)) + ReduceCost(g, splits);
}

// The cheaper kernel by the estimates above: columns per tile of the tensor-core kernel (0: the CUDA cores) and k splits.
// Both sides as measured (us, FFMA / tensor cores): [20, 600] x 200 14.7 / 13.4, [595, 450] x 150 12.8 / 12.6, [256, 1536]
// x 512 27 / 12.2 (4 k splits), [1500, 600] x 300 33 / 15.6, [400, 10000] x 200 84 / 36, [14474, 2048] x 512 1204 / 258;
// below one 64-wide k block the FFMA kernel is ahead.
struct Choice { int tile_n, splits; double us; };
Choice Choose(const GemmF32Args& g) {
  const long long tiles = static_cast<long long>((g.n + kTN - 1) / kTN) * ((g.m + kTM - 1) / kTM);
  const int sms = SmCount(), plain = PlainSplits(g, tiles, sms);
  Choice c{0, plain, PlainCost(g, tiles, plain, sms)};
  for (int tile : {128, 64})
    for (int z = 1; z <= 32 && g.k > 0; z *= 2) {
      if (z > 1 && (g.scratch_bytes == 0 || z > (g.k + 63) / 64 || static_cast<size_t>(z) * g.m * g.n * sizeof(float) > g.scratch_bytes)) break;
      const double us = SplitCost(g, tile, z, sms);
      if (us < c.us) c = {tile, z, us};
    }
  return c;
}

// The most k splits that Choose considers.
size_t MaxSplits(size_t k) {
  size_t z = 1;
  while (z < 32 && 2 * z <= (k + 63) / 64) z *= 2;
  return k >= 256 ? std::max(z, std::min<size_t>(16, k / 64)) : z;
}

int Check(const GemmF32Args& g) {
  CAVS_REQUIRE(g.m >= 0 && g.n >= 0 && g.k >= 0, CAVS_ERR_BAD_ARG, "gemm_f32: negative dimension");
  CAVS_REQUIRE(g.m == 0 || g.n == 0 || (g.a && g.b && g.c), CAVS_ERR_BAD_ARG, "gemm_f32: null pointer");
  return CAVS_OK;
}

int Run(const GemmF32Args& g_in, int tile_n, int splits, cudaStream_t stream) {
  GemmF32Args g = g_in;
  g.k_per_split = 0;
  if (tile_n > 0) {
    if (int rc = GemmF32Split(g, tile_n, &splits, stream)) return rc;
  } else {
    dim3 grid((g.n + kTN - 1) / kTN, (g.m + kTM - 1) / kTM);
    if (splits > 1) {
      g.k_per_split = ((g.k + splits - 1) / splits + kTK - 1) / kTK * kTK;
      splits = (g.k + g.k_per_split - 1) / g.k_per_split;
      grid.z = splits;
    }
    GemmF32Kernel<<<grid, 256, 0, stream>>>(g);
    CAVS_LAUNCH_CHECK("gemm_f32");
  }
  if (splits > 1) {
    CAVS_CUDA(LaunchChained(GemmF32Reduce, dim3(GridForElems(static_cast<size_t>(g.m) * g.n, 256)), dim3(256), 0, stream, g_in.c,
                            g_in.ldc, static_cast<const float*>(g.scratch), g.m, g.n, splits, g_in.accumulate ? 1 : 0));
    CAVS_LAUNCH_CHECK("gemm_f32 split reduce");
  }
  return CAVS_OK;
}

}  // namespace

size_t GemmF32ScratchBytes(size_t m, size_t n, size_t k) { return MaxSplits(k) > 1 ? MaxSplits(k) * m * n * sizeof(float) : 0; }
size_t GemmF32ScratchCap() { return static_cast<size_t>(2) * SmCount() * 128 * 128 * sizeof(float); }

double GemmF32Us(int m, int n, int k, size_t scratch_bytes) {
  GemmF32Args g;
  g.m = m; g.n = n; g.k = k;
  g.scratch_bytes = scratch_bytes;
  return Choose(g).us;
}

int GemmF32(const GemmF32Args& g_in, cudaStream_t stream) {
  GemmF32Args g = g_in;
  if (int rc = Check(g)) return rc;
  if (g.m == 0 || g.n == 0) return CAVS_OK;
  if (g.scratch == nullptr) g.scratch_bytes = 0;
  const Choice c = Choose(g);
  return Run(g, c.tile_n, c.splits, stream);
}

int GemmF32Tiled(const GemmF32Args& g, int tile_n, int splits, cudaStream_t stream) {
  if (int rc = Check(g)) return rc;
  CAVS_REQUIRE(tile_n == 0 || ((tile_n == 64 || tile_n == 128) && g.k > 0), CAVS_ERR_BAD_ARG,
               "gemm_f32_tiled: tile_n must be 0, or 64 or 128 with k >= 1");
  CAVS_REQUIRE(splits == 1 || (splits > 1 && g.k > 0 && g.scratch != nullptr && static_cast<size_t>(splits) * g.m * g.n * sizeof(float) <= g.scratch_bytes),
               CAVS_ERR_BAD_ARG, "gemm_f32_tiled: k splits need scratch for splits x m x n floats");
  if (g.m == 0 || g.n == 0) return CAVS_OK;
  return Run(g, tile_n, splits, stream);
}

}  // namespace cavs_b200

extern "C" int cavs_gemm_f32(float* c, long long ldc, int accumulate, const float* a, long long a_row_stride,
                             long long a_col_stride, const float* b, long long b_row_stride, long long b_col_stride, int m,
                             int n, int k, void* stream) {
  cavs_b200::GemmF32Args g;
  g.c = c; g.ldc = ldc; g.accumulate = accumulate;
  g.a = a; g.a_rs = a_row_stride; g.a_cs = a_col_stride;
  g.b = b; g.b_rs = b_row_stride; g.b_cs = b_col_stride;
  g.m = m; g.n = n; g.k = k;
  return cavs_b200::GemmF32(g, static_cast<cudaStream_t>(stream));
}

extern "C" int cavs_gemm_f32_tiled(float* c, long long ldc, int accumulate, const float* a, long long a_row_stride,
                                   long long a_col_stride, const float* b, long long b_row_stride, long long b_col_stride, int m,
                                   int n, int k, int tile_n, int splits, int withhold, float* scratch, size_t scratch_bytes, void* stream) {
  cavs_b200::GemmF32Args g;
  g.c = c; g.ldc = ldc; g.accumulate = accumulate;
  g.a = a; g.a_rs = a_row_stride; g.a_cs = a_col_stride;
  g.b = b; g.b_rs = b_row_stride; g.b_cs = b_col_stride;
  g.m = m; g.n = n; g.k = k;
  g.scratch = scratch; g.scratch_bytes = scratch_bytes; g.withhold = withhold;
  return cavs_b200::GemmF32Tiled(g, tile_n, splits, static_cast<cudaStream_t>(stream));
}

extern "C" int cavs_gemm_f32_choice(int m, int n, int k, size_t scratch_bytes, int* tile_n, int* splits) {
  using namespace cavs_b200;
  CAVS_REQUIRE(m > 0 && n > 0 && k >= 0 && tile_n && splits, CAVS_ERR_BAD_ARG, "gemm_f32_choice: bad argument");
  GemmF32Args g;
  g.m = m; g.n = n; g.k = k;
  g.scratch_bytes = scratch_bytes;
  const Choice c = Choose(g);
  *tile_n = c.tile_n;
  *splits = c.splits;
  return CAVS_OK;
}
