// The narrow levels of the fp32 Tree-LSTM in one launch per direction: a persistent grid walks the levels, a bounded
// grid barrier between them.
//
// Level by level a forward level is four launches (child gather, two products, cell) and a backward level four more
// (cell gradient, two products, scatter), each with its launch, its fill and its own round trip to memory: 25-35 us
// per level and direction however few rows it has.  Here a CTA keeps its slice of the recurrent weights in shared memory
// for all levels, a tile of rows is gathered, multiplied, finished and stored by the CTA that owns its columns, and a
// level costs a barrier, a few dependent round trips to L2 and its arithmetic (FFMA in fp32, k ascending within a
// k slice).  Twenty rows, H = 200, one child slot: 25 -> 4.9 us forward, 27 -> 8 us backward.  Wide levels stay with the tensor-core products: the multiply-adds here are bound by shared-memory reads (146
// rows, H = 512: 20 us forward, 53 backward).
//
// Forward: CTA (column group, row group) owns w hidden units with all four gates; a warp's lanes are 8 rows x 4 units,
// each thread RPT rows of one unit, and the k range is cut over the warps that share units (summed in order through
// shared memory).  Backward: one phase forms the gate gradients (threads own columns, so the bias gradient stays in
// registers), a barrier, one phase multiplies them with the transposed weights; w output columns per CTA.
// Rows are read with L1 bypassed: lines at row boundaries are shared with rows written in a later level.
#include <algorithm>
#include <cstdint>

#include "abi_common.h"
#include "kernels/cell.h"
#include "kernels/launch.h"
#include "kernels/narrow.cuh"
#include "kernels/narrow.h"

namespace cavs_b200 {
namespace {

using namespace narrow;

template <int K> constexpr int TileRows() { return K <= 2 ? 32 : 16; }

__host__ __device__ inline int Pad4(int x) { return (x + 3) & ~3; }
// Row pitch with which eight consecutive rows start in eight different groups of four banks.
__host__ __device__ inline int Pitch(int x) { return ((x + 31) & ~31) + 4; }

// rows x H floats (row r at src(r), nullptr: zeros) into dst (row pitch p), columns up to Pad4(H) zeroed, through registers
// with L1 bypassed, eight loads in flight per thread: widths whose rows are no whole 16-byte words.
template <int V, typename F>
__device__ __forceinline__ void LoadRows(float* dst, int p, int rows, int H, F src) {
  const int hv = Pad4(H) / V, tpr = hv <= 32 ? 32 : hv <= 64 ? 64 : 128, lane = threadIdx.x & (tpr - 1), step = kThreads / tpr;
  constexpr int kBatch = 8;
  for (int r0 = threadIdx.x / tpr; r0 < rows; r0 += step * kBatch)
    for (int j = lane; j < hv; j += tpr) {
      float v[kBatch][V];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int r = r0 + u * step;
        const float* s = r < rows && j * V < H ? src(r) : nullptr;
#pragma unroll
        for (int e = 0; e < V; ++e) v[u][e] = 0.0f;
        if (s != nullptr) {
          if constexpr (V == 2) { const float2 t = __ldcg(reinterpret_cast<const float2*>(s) + j); v[u][0] = t.x; v[u][1] = t.y; }
          else v[u][0] = __ldcg(s + j);
        }
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
        if (r0 + u * step < rows) {
#pragma unroll
          for (int e = 0; e < V; ++e) dst[(r0 + u * step) * p + j * V + e] = v[u][e];
        }
    }
}
// The same by one warp with bulk copies (H a multiple of 4), lane r taking row r of up to 32; arrives once on the buffer.
template <int kBuffers, typename F>
__device__ __forceinline__ void CopyRows(BulkRows<kBuffers>& ring, int buf, float* dst, int p, int rows, int H, F src) {
  const int lane = threadIdx.x & 31;
  const float* s = lane < rows ? src(lane) : nullptr;
  unsigned empty = __ballot_sync(0xffffffffu, lane < rows && s == nullptr);
  for (; empty != 0; empty &= empty - 1)   // no child there: zeros
    for (int j = lane * 4; j < H; j += 128) *reinterpret_cast<float4*>(dst + (__ffs(empty) - 1) * p + j) = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();
  ring.Copy(buf, static_cast<uint32_t>(__cvta_generic_to_shared(dst)), p * 4, s, H * 4);
}

// ---- forward ----
template <int K, int RPT>
__device__ __forceinline__ void FwdProducts(const float* At, int p, const float4* Ub, int w, int unit, int k4_begin, int k4_end, float* red,
                                            int lane) {
  constexpr int TR = TileRows<K>(), G = 3 + K;
  float acc[RPT][G];
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int g = 0; g < G; ++g) acc[r][g] = 0.0f;
  const float* a0 = At + (lane >> 2) * p;
#pragma unroll 2
  for (int k4 = k4_begin; k4 < k4_end; ++k4) {
    float4 b[4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) b[kk] = Ub[(k4 * 4 + kk) * w + unit];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      float h[K][4], s[4];
#pragma unroll
      for (int c = 0; c < K; ++c) {
        const float4 t = *reinterpret_cast<const float4*>(a0 + (c * TR + r * 8) * p + k4 * 4);
        h[c][0] = t.x; h[c][1] = t.y; h[c][2] = t.z; h[c][3] = t.w;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) s[kk] = c == 0 ? h[c][kk] : s[kk] + h[c][kk];
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        acc[r][0] = fmaf(s[kk], b[kk].x, acc[r][0]);
        acc[r][1] = fmaf(s[kk], b[kk].y, acc[r][1]);
        acc[r][2] = fmaf(s[kk], b[kk].z, acc[r][2]);
#pragma unroll
        for (int c = 0; c < K; ++c) acc[r][3 + c] = fmaf(h[c][kk], b[kk].w, acc[r][3 + c]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int g = 0; g < G; ++g) red[(g * TR + (lane >> 2) + r * 8) * w + unit] = acc[r][g];
}

template <int K, int V>
__global__ void __launch_bounds__(kThreads, 1) NarrowForward(const NarrowForwardArgs a) {
  constexpr int TR = TileRows<K>(), G = 3 + K;
  extern __shared__ __align__(16) float smem[];
  __shared__ int s_child[2][K][TR];
  const int H = a.H, w = a.w, hk = Pad4(H), p = Pitch(hk);
  float4* Ub = reinterpret_cast<float4*>(smem);                 // [hk][w]: i, o, u, f columns of a unit
  float* At0 = smem + static_cast<size_t>(hk) * w * 4;           // [buffers][K][TR][p]
  float* red = At0 + a.buffers * K * TR * p;                                  // [k slices][G][TR][w]
  const int cg = blockIdx.x % a.col_groups, rg = blockIdx.x / a.col_groups, j0 = cg * w;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit_warps = w / 4, slices = kWarps / unit_warps;
  const int unit = (warp % unit_warps) * 4 + (lane & 3), slice = warp / unit_warps;
  const int k4_per = (hk / 4 + slices - 1) / slices, k4_begin = min(hk / 4, slice * k4_per), k4_end = min(hk / 4, k4_begin + k4_per);
  for (int i = threadIdx.x; i < hk * w; i += kThreads) {
    const int k = i / w, j = j0 + i % w;
    const bool in = k < H && j < H;
    const float* u = static_cast<const float*>(a.U_iou) + static_cast<size_t>(k) * 3 * H + j;
    Ub[i] = in ? make_float4(u[0], u[H], u[2 * H], static_cast<const float*>(a.U_f)[static_cast<size_t>(k) * H + j]) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // the pair (row of a tile, unit) that this thread finishes
  const int prow = threadIdx.x / w, pj = j0 + threadIdx.x % w;
  const bool pair = prow < TR && pj < H;
  float bi = 0.f, bf = 0.f, bu = 0.f, bo = 0.f;
  if (pair) { bi = a.bias[pj]; bf = a.bias[H + pj]; bu = a.bias[2 * H + pj]; bo = a.bias[3 * H + pj]; }

  __shared__ uint64_t s_full[2];
  BulkRows<2> ring;
  ring.Init(s_full, K);
  int off = __ldg(a.level_off + a.level_begin), end = __ldg(a.level_off + a.level_begin + 1);
  unsigned barrier = 0;
  // What the next tile needs beside the previous level's states is requested before the barrier.
  int child = -1;
  float in[4] = {};
  auto prefetch = [&](int off_, int end_, int tile) {
    child = -1;
    const int t = off_ + tile * TR + static_cast<int>(threadIdx.x) % TR;
    if (threadIdx.x < K * TR && t < end_) child = __ldg(a.child + static_cast<size_t>(threadIdx.x / TR) * a.n_total + t);
    const int tp = off_ + tile * TR + prow;
    if (pair && tp < end_) {
      const float* x = static_cast<const float*>(a.A) + static_cast<size_t>(a.a_row ? __ldg(a.a_row + tp) : tp) * 4 * H + pj;
#pragma unroll
      for (int g = 0; g < 4; ++g) in[g] = __ldg(x + g * H);
    }
  };
  prefetch(off, end, rg);
  for (int l = a.level_begin; l < a.level_end; ++l) {
    const int next_end = l + 1 < a.level_end ? __ldg(a.level_off + l + 2) : end;
    const int tiles = (end - off + TR - 1) / TR;
    // Rows of tile `tile` into buffer `buf`, children from s_child[buf].
    auto load_rows = [&](int tile, int buf) {
      const int live = min(TR, (end - off - tile * TR + 7) & ~7);   // whole groups of eight rows
#pragma unroll
      for (int c = 0; c < K; ++c) {
        auto row = [&](int r) -> const float* {
          const int ch = s_child[buf][c][r];
          return ch >= 0 ? a.state + static_cast<size_t>(ch) * 2 * H : nullptr;
        };
        if constexpr (V == 4) {
          if (warp == c) CopyRows(ring, buf, At0 + (buf * K + c) * TR * p, p, live, H, row);
        } else {
          LoadRows<V>(At0 + (buf * K + c) * TR * p, p, live, H, row);
        }
      }
    };
    int buf = 0;
    for (int tile = rg; tile < tiles; tile += a.row_groups, buf ^= 1) {
      const int t0 = off + tile * TR, rows = min(TR, end - t0), nbuf = a.buffers == 2 ? buf : 0;
      const bool more = tile + a.row_groups < tiles;
      if (tile == rg) {
        if (threadIdx.x < K * TR) s_child[0][threadIdx.x / TR][threadIdx.x % TR] = child;
        __syncthreads();
        load_rows(tile, 0);
      } else if (a.buffers == 1) {
        load_rows(tile, 0);
      }
      float c_in[K], x[4];
#pragma unroll
      for (int c = 0; c < K; ++c) c_in[c] = 0.0f;
#pragma unroll
      for (int g = 0; g < 4; ++g) x[g] = in[g];
      const int sc = a.buffers == 2 ? buf : 0;
      if (pair && prow < rows) {
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const int ch = s_child[sc][c][prow];
          if (ch >= 0) c_in[c] = __ldcg(a.state + static_cast<size_t>(ch) * 2 * H + H + pj);
        }
      }
      if (more) {
        prefetch(off, end, tile + a.row_groups);
        if (a.buffers == 2 && threadIdx.x < K * TR) s_child[buf ^ 1][threadIdx.x / TR][threadIdx.x % TR] = child;
      }
      if constexpr (V == 4) ring.Wait(nbuf, a.status);
      __syncthreads();
      if (more && a.buffers == 2) load_rows(tile + a.row_groups, buf ^ 1);   // arrives under this tile's products
      const float* At = At0 + nbuf * K * TR * p;
      float* my_red = red + slice * TR * w * G;
      if (rows <= 8) FwdProducts<K, 1>(At, p, Ub, w, unit, k4_begin, k4_end, my_red, lane);
      else if (rows <= 16 || TR == 16) FwdProducts<K, 2>(At, p, Ub, w, unit, k4_begin, k4_end, my_red, lane);
      else FwdProducts<K, TR / 8>(At, p, Ub, w, unit, k4_begin, k4_end, my_red, lane);
      __syncthreads();
      if (pair && prow < rows) {
        float z[G];
#pragma unroll
        for (int g = 0; g < G; ++g) z[g] = 0.0f;
#pragma unroll 4
        for (int s = 0; s < slices; ++s)
#pragma unroll
          for (int g = 0; g < G; ++g) z[g] += red[(s * G + g) * TR * w + threadIdx.x];
        const size_t t = t0 + prow;
        const float gi = Sigmoid<false>((x[0] + z[0]) + bi), go = Sigmoid<false>((x[1] + z[1]) + bo), gu = tanhf((x[2] + z[2]) + bu);
        float cc = gi * gu, sum = 0.0f;
        float* g = static_cast<float*>(a.gates) + t * G * H + pj;
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const float gf = Sigmoid<false>((x[3] + z[3 + c]) + bf);
          cc = cc + gf * c_in[c];
          g[(3 + c) * H] = gf;
          const float h = At[(c * TR + prow) * p + pj];
          sum = c == 0 ? h : sum + h;
          static_cast<float*>(a.HK)[(t * K + c) * H + pj] = h;
        }
        static_cast<float*>(a.S)[t * H + pj] = sum;
        g[0] = gi; g[H] = go; g[2 * H] = gu;
        a.state[t * 2 * H + pj] = go * tanhf(cc);
        a.state[t * 2 * H + H + pj] = cc;
      }
      if (more) {
        if (a.buffers == 1 && threadIdx.x < K * TR) s_child[0][threadIdx.x / TR][threadIdx.x % TR] = child;
        __syncthreads();   // readers of At and red are done
      }
    }
    off = end; end = next_end;
    if (l + 1 < a.level_end) {
      GridArrive(a.barrier);
      prefetch(off, end, rg);
      if (!GridWait(a.barrier, ++barrier * gridDim.x + a.withhold, a.status)) { ring.Drain(); return; }
    }
  }
  ring.Drain();
}

// ---- backward ----
template <int RPT, int NPT>
__device__ __forceinline__ void BwdProducts(float (&acc)[RPT][NPT], const float* At, int p, const float* Wt, int pw, int k4_begin, int k4_end,
                                            int lane) {
  const float* a0 = At + (lane >> 2) * p;
#pragma unroll 2
  for (int k4 = k4_begin; k4 < k4_end; ++k4) {
    float4 b[NPT];
#pragma unroll
    for (int n = 0; n < NPT; ++n) b[n] = *reinterpret_cast<const float4*>(Wt + n * 4 * pw + k4 * 4);
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const float4 x = *reinterpret_cast<const float4*>(a0 + r * 8 * p + k4 * 4);
#pragma unroll
      for (int n = 0; n < NPT; ++n) {
        acc[r][n] = fmaf(x.x, b[n].x, acc[r][n]);
        acc[r][n] = fmaf(x.y, b[n].y, acc[r][n]);
        acc[r][n] = fmaf(x.z, b[n].z, acc[r][n]);
        acc[r][n] = fmaf(x.w, b[n].w, acc[r][n]);
      }
    }
  }
}

// One tile of the second phase: d(h) of the children of rows [t0, t0 + rows), this CTA's columns.
template <int K, int V, int NPT, int RPT>
__device__ __forceinline__ void BwdTile(const NarrowBackwardArgs& a, const float* Wt, int pw, float* At, int p, float* red, BulkRows<3 + K>& ring, int t0, int rows, int n0,
                                        int unit, int slice, int slices, int k4_begin, int k4_end) {
  constexpr int TR = TileRows<K>(), G = 3 + K;
  const int H = a.H, w = a.w, hk = Pad4(H), lane = threadIdx.x & 31;
  const int prow = threadIdx.x / w, col = n0 + threadIdx.x % w;
  const bool pair = prow < rows && col < H;
  int chn[K];
#pragma unroll
  for (int c = 0; c < K; ++c) chn[c] = pair ? __ldg(a.child + static_cast<size_t>(c) * a.n_total + t0 + prow) : -1;
  float ds[RPT][NPT], dq[K][RPT][NPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int n = 0; n < NPT; ++n) {
      ds[r][n] = 0.0f;
#pragma unroll
      for (int c = 0; c < K; ++c) dq[c][r][n] = 0.0f;
    }
  // Vectors zi, zo, zu, zf_0.. pass through a ring of buffers: as many as fit are requested ahead of their products.
  auto load = [&](int q) {
    auto row = [&](int r) -> const float* {
      if (r >= rows) return nullptr;
      const size_t t = t0 + r;
      return q < 3 ? static_cast<const float*>(a.dA) + t * 4 * H + q * H : static_cast<const float*>(a.ZF) + (t * K + q - 3) * H;
    };
    float* dst = At + (q % a.buffers) * TR * p;
    if constexpr (V == 4) {
      if (static_cast<int>(threadIdx.x >> 5) == q) CopyRows(ring, q % a.buffers, dst, p, rows, H, row);
    } else {
      LoadRows<V>(dst, p, RPT * 8, H, row);
    }
  };
  __syncthreads();   // readers of the buffers and of the sums are done
  const int ahead = min(a.buffers, G);
  for (int q = 0; q < ahead; ++q) load(q);
#pragma unroll
  for (int q = 0; q < G; ++q) {
    if constexpr (V == 4) ring.Wait(q % a.buffers, a.status);
    else __syncthreads();
    const float* buf = At + (q % a.buffers) * TR * p;
    const float* wt = Wt + unit * pw + min(q, 3) * hk;
    if (q < 3) BwdProducts<RPT, NPT>(ds, buf, p, wt, pw, k4_begin, k4_end, lane);
    else BwdProducts<RPT, NPT>(dq[q < 3 ? 0 : q - 3], buf, p, wt, pw, k4_begin, k4_end, lane);
    if (q + a.buffers < G) {
      __syncthreads();
      load(q + a.buffers);
    }
  }
  float* my_red = red + slice * TR * w * (1 + K);
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int n = 0; n < NPT; ++n) {
      float* x = my_red + ((lane >> 2) + r * 8) * w + unit + n * 4;
      x[0] = ds[r][n];
#pragma unroll
      for (int c = 0; c < K; ++c) x[(1 + c) * TR * w] = dq[c][r][n];
    }
  __syncthreads();
  if (pair) {
    float z[1 + K];
#pragma unroll
    for (int c = 0; c <= K; ++c) z[c] = 0.0f;
#pragma unroll 4
    for (int s = 0; s < slices; ++s)
#pragma unroll
      for (int c = 0; c <= K; ++c) z[c] += red[(s * (1 + K) + c) * TR * w + threadIdx.x];
#pragma unroll
    for (int c = 0; c < K; ++c)
      if (chn[c] >= 0) a.mailbox[static_cast<size_t>(chn[c]) * 2 * H + col] = z[0] + z[1 + c];
  }
}

template <int K, int V, int NPT>
__global__ void __launch_bounds__(kThreads, 1) NarrowBackward(const NarrowBackwardArgs a) {
  constexpr int TR = TileRows<K>();
  extern __shared__ __align__(16) float smem[];
  const int H = a.H, w = a.w, hk = Pad4(H), p = Pitch(hk), pw = Pitch(4 * hk);
  float* Wt = smem;                        // [w][pw]: row n of U_iou (three blocks) and U_f, each block padded to hk
  float* At = Wt + static_cast<size_t>(w) * pw;   // [buffers][TR][p]
  float* red = At + static_cast<size_t>(a.buffers) * TR * p;   // [k slices][1 + K][TR][w]
  const int cg = blockIdx.x % a.col_groups, rg = blockIdx.x / a.col_groups, n0 = cg * w;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit_warps = w / (4 * NPT), slices = kWarps / unit_warps;
  const int unit = (warp % unit_warps) * 4 * NPT + (lane & 3), slice = warp / unit_warps;
  const int k4_per = (hk / 4 + slices - 1) / slices, k4_begin = min(hk / 4, slice * k4_per), k4_end = min(hk / 4, k4_begin + k4_per);
  for (int n = 0; n < w; ++n)
    for (int i = threadIdx.x; i < 4 * hk; i += kThreads) {
      const int q = i / hk, k = i - q * hk, col = n0 + n;
      float v = 0.0f;
      if (col < H && k < H) v = q < 3 ? static_cast<const float*>(a.U_iou)[static_cast<size_t>(col) * 3 * H + q * H + k] : static_cast<const float*>(a.U_f)[static_cast<size_t>(col) * H + k];
      Wt[n * pw + i] = v;
    }
  GateGradients<K, float, float> gg(a);
  __shared__ uint64_t s_full[3 + K];
  BulkRows<3 + K> ring;
  ring.Init(s_full, 1);
  __syncthreads();

  int end = __ldg(a.level_off + a.level_end), off = __ldg(a.level_off + a.level_end - 1);
  unsigned barrier = 0;
  gg.Request(a, off, end);
  for (int l = a.level_end - 1; l >= a.level_begin; --l) {
    const int next_off = l > a.level_begin ? __ldg(a.level_off + l - 1) : 0;
    gg.Level(a, off, end);
    GridArrive(a.barrier);
    if (l > a.level_begin) gg.Request(a, next_off, off);   // only the mailbox rows are not complete yet
    if (!GridWait(a.barrier, ++barrier * gridDim.x + a.withhold, a.status)) { ring.Drain(); return; }
    const int tiles = (end - off + TR - 1) / TR;
    for (int tile = rg; tile < tiles; tile += a.row_groups) {
      const int t0 = off + tile * TR, rows = min(TR, end - t0);
      if (rows <= 8) BwdTile<K, V, NPT, 1>(a, Wt, pw, At, p, red, ring, t0, rows, n0, unit, slice, slices, k4_begin, k4_end);
      else BwdTile<K, V, NPT, TR / 8>(a, Wt, pw, At, p, red, ring, t0, rows, n0, unit, slice, slices, k4_begin, k4_end);
    }
    end = off; off = next_off;
    if (gg.local) {
      __syncthreads();   // the next level's rows of these columns were written by this CTA
    } else if (l > a.level_begin) {
      GridArrive(a.barrier);
      if (!GridWait(a.barrier, ++barrier * gridDim.x + a.withhold, a.status)) { ring.Drain(); return; }
    }
  }
  gg.FoldSums(a, red);
  ring.Drain();
}

size_t ForwardSmem(int H, int K, int w, int buffers) {
  const int hk = Pad4(H), tr = K <= 2 ? 32 : 16, slices = kWarps / (w / 4);
  return sizeof(float) * (static_cast<size_t>(hk) * w * 4 + static_cast<size_t>(buffers) * K * tr * Pitch(hk) + static_cast<size_t>(slices) * tr * w * (3 + K));
}
int BackwardNpt(int w) { return w >= 8 ? 2 : 1; }
size_t BackwardSmem(int H, int K, int w, int buffers) {
  const int hk = Pad4(H), tr = K <= 2 ? 32 : 16, slices = kWarps / (w / (4 * BackwardNpt(w)));
  const size_t red = std::max(static_cast<size_t>(slices) * tr * w * (1 + K), static_cast<size_t>(4) * kThreads);
  return sizeof(float) * (static_cast<size_t>(w) * Pitch(4 * hk) + static_cast<size_t>(buffers) * tr * Pitch(hk) + red);
}

template <int K, int V>
int ForwardKV(const NarrowForwardArgs& a, int grid, size_t smem, cudaStream_t st) { return LaunchCooperative<NarrowForward<K, V>>(a, grid, smem, st); }
template <int K>
int ForwardK(const NarrowForwardArgs& a, int grid, size_t smem, cudaStream_t st) {
  return a.H % 4 == 0 ? ForwardKV<K, 4>(a, grid, smem, st) : a.H % 2 == 0 ? ForwardKV<K, 2>(a, grid, smem, st) : ForwardKV<K, 1>(a, grid, smem, st);
}
template <int K, int V>
int BackwardKV(const NarrowBackwardArgs& a, int grid, size_t smem, cudaStream_t st) {
  return BackwardNpt(a.w) == 2 ? LaunchCooperative<NarrowBackward<K, V, 2>>(a, grid, smem, st) : LaunchCooperative<NarrowBackward<K, V, 1>>(a, grid, smem, st);
}
template <int K>
int BackwardK(const NarrowBackwardArgs& a, int grid, size_t smem, cudaStream_t st) {
  return a.H % 4 == 0 ? BackwardKV<K, 4>(a, grid, smem, st) : a.H % 2 == 0 ? BackwardKV<K, 2>(a, grid, smem, st) : BackwardKV<K, 1>(a, grid, smem, st);
}

}  // namespace

NarrowPlan PlanNarrowF32(int H, int K, int rows, bool backward) {
  NarrowPlan best;
  const int tr = K <= 2 ? 32 : 16;
  const int tiles = (rows + tr - 1) / tr, sms = SmCount();
  double best_cost = 0.0;
  for (int w : {4, 8, 16})
   for (int groups : {1, 2}) {   // one row group, or as many as fit
    const int cols = (H + w - 1) / w;
    if (cols > sms) continue;
    NarrowPlan p;
    p.w = w;
    p.col_groups = cols;
    p.row_groups = groups == 1 ? 1 : std::min(sms / cols, tiles);
    p.buffers = 3 + K;
    if (backward) {
      while (p.buffers > 0 && BackwardSmem(H, K, w, p.buffers) > kMaxSmem) --p.buffers;
      if (p.buffers == 0) continue;
      p.smem = BackwardSmem(H, K, w, p.buffers);
    } else {
      p.buffers = tiles > p.row_groups && ForwardSmem(H, K, w, 2) <= kMaxSmem ? 2 : 1;
      p.smem = ForwardSmem(H, K, w, p.buffers);
      if (p.smem > kMaxSmem) continue;
    }
    // us per level: row tiles in sequence, each its fused multiply-adds (bound by shared-memory reads: 11-30 % of the
    // pipe as measured, the more the more columns a thread has) and, unless a second buffer lets it arrive under the
    // previous tile's, its gather
    const double rate = backward ? (w >= 8 ? 0.15 : 0.11) : (w >= 8 ? 0.28 : 0.2);
    const double load = backward ? 0.5 * (3 + K) : 1.0, work = static_cast<double>(tr) * w * H * (3 + K) / (128.0 * rate * 1900.0);
    const int mine = (tiles + p.row_groups - 1) / p.row_groups;
    // (backward: the second barrier, which one row group does without)
    const double cost = (p.buffers > 1 ? load + mine * std::max(work, 0.6 * load) : mine * (load + work)) + (backward && p.row_groups > 1 ? 2.5 : 0.0);
    if (best.w == 0 || cost < best_cost) { best = p; best_cost = cost; }
  }
  return best;
}

// Fitted to what levels of 1 to 8192 rows took inside chains of such levels, H = 32 .. 512 and one, two and four child slots
// (root mean square error 11 % forward, 13 % backward; 10 % where the per-level launches take as long).  A CTA takes every
// row_groups-th row tile; a level costs its barrier and round trips, each tile in sequence, the rows and multiply-adds of
// a CTA, rows of no whole 16-byte words (read through registers), and the grid's rows together; backward also the second
// barrier, a thread's rows of gate gradients and the vectors that find no buffer.
double NarrowLevelUsF32(const NarrowPlan& p, int H, int K, int rows, bool backward) {
  const int tr = K <= 2 ? 32 : 16, vectors = 3 + K, read = backward ? vectors : K, tiles = (rows + tr - 1) / tr;
  const int mine = (tiles + p.row_groups - 1) / p.row_groups;
  const double mb = 4e-6 * std::min(rows, mine * tr) * H * read, mac = 1e-6 * mine * tr * p.w * H * vectors;
  const double runs = (H % 4 == 0 ? 0 : H % 2 == 0 ? 1 : 2) * 1e-3 * mine * read * H, all = 1e-3 * rows * vectors;
  if (!backward) return 1.35 + mine * (1.97 + 0.185 * K) + 22.1 * mb + (p.w == 4 ? 4.6 : 7.4) * mac + 3.0 * runs + 0.14 * all;
  const bool local = p.row_groups == 1;
  const int cols = local ? p.w : narrow::kColBlock, strips = local ? 1 : std::max(1, p.col_groups * p.row_groups / ((H + cols - 1) / cols));
  const int step = strips * (kThreads / cols);
  return 0.33 + mine * (3.3 + 0.48 * K) + 11.3 * mb + (p.w == 4 ? 1.15 : 8.8) * mac + 3.85 * runs + 1.04 * all + (local ? 0.0 : 2.5) +
         1.3 * ((rows + step - 1) / step) + 0.97 * mine * std::max(0, vectors - p.buffers);
}

int LaunchNarrowForwardF32(const NarrowPlan& plan, NarrowForwardArgs a, int K, cudaStream_t st) {
  a.w = plan.w; a.col_groups = plan.col_groups; a.row_groups = plan.row_groups; a.buffers = plan.buffers;
  const int grid = plan.col_groups * plan.row_groups;
  switch (K) {
    case 1: return ForwardK<1>(a, grid, plan.smem, st);
    case 2: return ForwardK<2>(a, grid, plan.smem, st);
    case 3: return ForwardK<3>(a, grid, plan.smem, st);
    default: return ForwardK<4>(a, grid, plan.smem, st);
  }
}

int LaunchNarrowBackwardF32(const NarrowPlan& plan, NarrowBackwardArgs a, int K, cudaStream_t st) {
  a.w = plan.w; a.col_groups = plan.col_groups; a.row_groups = plan.row_groups; a.buffers = plan.buffers;
  const int grid = plan.col_groups * plan.row_groups;
  switch (K) {
    case 1: return BackwardK<1>(a, grid, plan.smem, st);
    case 2: return BackwardK<2>(a, grid, plan.smem, st);
    case 3: return BackwardK<3>(a, grid, plan.smem, st);
    default: return BackwardK<4>(a, grid, plan.smem, st);
  }
}

}  // namespace cavs_b200
