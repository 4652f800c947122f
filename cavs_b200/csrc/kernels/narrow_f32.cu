// The narrow levels of the fp32 Tree-LSTM in one launch per direction: a persistent grid walks the levels, a bounded
// grid barrier between them.
//
// Level by level a forward level is four launches (child gather, two products, cell) and a backward level four more
// (cell gradient, two products, scatter), each with its launch, its fill and its own round trip to memory: 25-35 us
// per level and direction however few rows it has, while the arithmetic of a level of 64 rows and H = 512 takes
// 2 us of the chip.  Here a CTA keeps its slice of the recurrent weights in shared memory for all levels, a tile of
// rows is gathered, multiplied, finished and stored by the CTA that owns its columns, and a level costs a barrier
// and its arithmetic (FFMA in fp32, k ascending within a k slice).
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
#include "kernels/narrow.h"

namespace cavs_b200 {
namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr unsigned kBarrierPolls = 1u << 19;   // about half a second
template <int K> constexpr int TileRows() { return K <= 2 ? 32 : 16; }

__host__ __device__ inline int Pad4(int x) { return (x + 3) & ~3; }
// Row pitch with which eight consecutive rows start in eight different groups of four banks.
__host__ __device__ inline int Pitch(int x) { return ((x + 31) & ~31) + 4; }

__device__ __forceinline__ float SigmoidF(float x) { return 1.0f / (1.0f + expf(-x)); }

// All CTAs of the grid (launched cooperatively) arrive; false, and *status raised, if that takes too long.
__device__ __forceinline__ bool GridSync(unsigned* counter, unsigned target, int* status) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    int ok = 0;
    for (unsigned it = 0; it < kBarrierPolls; ++it) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if (v >= target) { ok = 1; break; }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    if (!ok) atomicExch(status, 1);
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// rows x H floats (row r at src(r), nullptr: zeros) into dst (row pitch p), columns up to Pad4(H) zeroed.
template <int V, typename F>
__device__ __forceinline__ void LoadRows(float* dst, int p, int rows, int H, F src) {
  const int hv = Pad4(H) / V;
#pragma unroll 4
  for (int i = threadIdx.x; i < rows * hv; i += kThreads) {
    const int r = i / hv, j = (i - r * hv) * V;
    const float* s = src(r);
    float v[V];
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = 0.0f;
    if (s != nullptr && j < H) {
      if constexpr (V == 4) { const float4 t = __ldcg(reinterpret_cast<const float4*>(s + j)); v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; }
      else if constexpr (V == 2) { const float2 t = __ldcg(reinterpret_cast<const float2*>(s + j)); v[0] = t.x; v[1] = t.y; }
      else v[0] = __ldcg(s + j);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) dst[r * p + j + e] = v[e];
  }
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
    for (int g = 0; g < G; ++g) red[(((lane >> 2) + r * 8) * w + unit) * G + g] = acc[r][g];
}

template <int K, int V>
__global__ void __launch_bounds__(kThreads, 1) NarrowForward(const NarrowForwardArgs a) {
  constexpr int TR = TileRows<K>(), G = 3 + K;
  extern __shared__ __align__(16) float smem[];
  __shared__ int s_child[K][TR];
  const int H = a.H, w = a.w, hk = Pad4(H), p = Pitch(hk);
  float4* Ub = reinterpret_cast<float4*>(smem);                 // [hk][w]: i, o, u, f columns of a unit
  float* At = smem + static_cast<size_t>(hk) * w * 4;            // [K][TR][p]
  float* red = At + K * TR * p;                                  // [k slices][TR][w][G]
  const int cg = blockIdx.x % a.col_groups, rg = blockIdx.x / a.col_groups, j0 = cg * w;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit_warps = w / 4, slices = kWarps / unit_warps;
  const int unit = (warp % unit_warps) * 4 + (lane & 3), slice = warp / unit_warps;
  const int k4_per = (hk / 4 + slices - 1) / slices, k4_begin = min(hk / 4, slice * k4_per), k4_end = min(hk / 4, k4_begin + k4_per);
  for (int i = threadIdx.x; i < hk * w; i += kThreads) {
    const int k = i / w, j = j0 + i % w;
    const bool in = k < H && j < H;
    const float* u = a.U_iou + static_cast<size_t>(k) * 3 * H + j;
    Ub[i] = in ? make_float4(u[0], u[H], u[2 * H], a.U_f[static_cast<size_t>(k) * H + j]) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // the pair (row of a tile, unit) that this thread finishes
  const int prow = threadIdx.x / w, pj = j0 + threadIdx.x % w;
  const bool pair = prow < TR && pj < H;
  float bi = 0.f, bf = 0.f, bu = 0.f, bo = 0.f;
  if (pair) { bi = a.bias[pj]; bf = a.bias[H + pj]; bu = a.bias[2 * H + pj]; bo = a.bias[3 * H + pj]; }

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
      const float* x = a.A + static_cast<size_t>(a.a_row ? __ldg(a.a_row + tp) : tp) * 4 * H + pj;
#pragma unroll
      for (int g = 0; g < 4; ++g) in[g] = __ldg(x + g * H);
    }
  };
  prefetch(off, end, rg);
  for (int l = a.level_begin; l < a.level_end; ++l) {
    const int next_end = l + 1 < a.level_end ? __ldg(a.level_off + l + 2) : end;
    const int tiles = (end - off + TR - 1) / TR;
    for (int tile = rg; tile < tiles; tile += a.row_groups) {
      const int t0 = off + tile * TR, rows = min(TR, end - t0);
      if (tile != rg) prefetch(off, end, tile);
      if (threadIdx.x < K * TR) s_child[threadIdx.x / TR][threadIdx.x % TR] = child;
      __syncthreads();   // also: the previous tile's readers of At and red are done
      float c_in[K];
#pragma unroll
      for (int c = 0; c < K; ++c) c_in[c] = 0.0f;
      if (pair && prow < rows) {
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const int ch = s_child[c][prow];
          if (ch >= 0) c_in[c] = __ldcg(a.state + static_cast<size_t>(ch) * 2 * H + H + pj);
        }
      }
      LoadRows<V>(At, p, K * TR, H, [&](int r) {
        const int ch = s_child[r / TR][r % TR];
        return ch >= 0 ? a.state + static_cast<size_t>(ch) * 2 * H : nullptr;
      });
      __syncthreads();
      float* my_red = red + slice * TR * w * G;
      if (rows <= 8) FwdProducts<K, 1>(At, p, Ub, w, unit, k4_begin, k4_end, my_red, lane);
      else if (rows <= 16 || TR == 16) FwdProducts<K, 2>(At, p, Ub, w, unit, k4_begin, k4_end, my_red, lane);
      else FwdProducts<K, TR / 8>(At, p, Ub, w, unit, k4_begin, k4_end, my_red, lane);
      __syncthreads();
      if (pair && prow < rows) {
        float z[G];
#pragma unroll
        for (int g = 0; g < G; ++g) z[g] = 0.0f;
        for (int s = 0; s < slices; ++s)
#pragma unroll
          for (int g = 0; g < G; ++g) z[g] += red[((s * TR + prow) * w + threadIdx.x % w) * G + g];
        const size_t t = t0 + prow;
        const float gi = SigmoidF((in[0] + z[0]) + bi), go = SigmoidF((in[1] + z[1]) + bo), gu = tanhf((in[2] + z[2]) + bu);
        float cc = gi * gu, sum = 0.0f;
        float* g = a.gates + t * G * H + pj;
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const float gf = SigmoidF((in[3] + z[3 + c]) + bf);
          cc = cc + gf * c_in[c];
          g[(3 + c) * H] = gf;
          const float h = At[(c * TR + prow) * p + pj];
          sum = c == 0 ? h : sum + h;
          a.HK[(t * K + c) * H + pj] = h;
        }
        a.S[t * H + pj] = sum;
        g[0] = gi; g[H] = go; g[2 * H] = gu;
        a.state[t * 2 * H + pj] = go * tanhf(cc);
        a.state[t * 2 * H + H + pj] = cc;
      }
      __syncthreads();
    }
    off = end; end = next_end;
    if (l + 1 < a.level_end) {
      prefetch(off, end, rg);
      if (!GridSync(a.barrier, ++barrier * gridDim.x, a.status)) return;
    }
  }
}

// ---- backward ----
constexpr int kColBlock = 64, kRowLanes = kThreads / kColBlock;

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

template <int K, int V, int NPT>
__global__ void __launch_bounds__(kThreads, 1) NarrowBackward(const NarrowBackwardArgs a) {
  constexpr int TR = TileRows<K>(), G = 3 + K, RPT = TR / 8;
  extern __shared__ __align__(16) float smem[];
  const int H = a.H, w = a.w, hk = Pad4(H), p = Pitch(hk), pw = Pitch(4 * hk);
  float* Wt = smem;                        // [w][pw]: row n of U_iou (three blocks) and U_f, each block padded to hk
  float* At = Wt + static_cast<size_t>(w) * pw;   // [buffers][TR][p]
  float* red = At + static_cast<size_t>(a.buffers) * TR * p;   // [k slices][TR][w][1 + K]
  const int cg = blockIdx.x % a.col_groups, rg = blockIdx.x / a.col_groups, n0 = cg * w;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit_warps = w / (4 * NPT), slices = kWarps / unit_warps;
  const int unit = (warp % unit_warps) * 4 * NPT + (lane & 3), slice = warp / unit_warps;
  const int k4_per = (hk / 4 + slices - 1) / slices, k4_begin = min(hk / 4, slice * k4_per), k4_end = min(hk / 4, k4_begin + k4_per);
  for (int i = threadIdx.x; i < w * 4 * hk; i += kThreads) {
    const int n = i / (4 * hk), q = i % (4 * hk) / hk, k = i % hk, col = n0 + n;
    float v = 0.0f;
    if (col < H && k < H) v = q < 3 ? a.U_iou[static_cast<size_t>(col) * 3 * H + q * H + k] : a.U_f[static_cast<size_t>(col) * H + k];
    Wt[n * pw + q * hk + k] = v;
  }
  // gate gradients: this thread's column and its rows
  const int col_blocks = (H + kColBlock - 1) / kColBlock, strips = max(1, static_cast<int>(gridDim.x) / col_blocks);
  const int j = (blockIdx.x % col_blocks) * kColBlock + threadIdx.x % kColBlock, strip = blockIdx.x / col_blocks;
  const bool owner = j < H && strip < strips;
  float sums[4] = {}, wc[kHeadDzPitch];
#pragma unroll
  for (int c = 0; c < kHeadDzPitch; ++c) wc[c] = owner && a.dz != nullptr && c < a.C ? a.Wc[static_cast<size_t>(c) * H + j] : 0.0f;
  __syncthreads();

  int end = __ldg(a.level_off + a.level_end), off = __ldg(a.level_off + a.level_end - 1);
  unsigned barrier = 0;
  for (int l = a.level_end - 1; l >= a.level_begin; --l) {
    const int next_off = l > a.level_begin ? __ldg(a.level_off + l - 1) : 0;
    if (owner) {
#pragma unroll 2
      for (int t_ = off + strip * kRowLanes + static_cast<int>(threadIdx.x) / kColBlock; t_ < end; t_ += strips * kRowLanes) {
        const size_t t = t_;
        const bool has_parent = __ldg(a.parent + t) >= 0;
        int ch[K], chs[K];
#pragma unroll
        for (int c = 0; c < K; ++c) {
          ch[c] = __ldg(a.child + static_cast<size_t>(c) * a.n_total + t);
          chs[c] = a.child_state ? __ldg(a.child_state + static_cast<size_t>(c) * a.n_total + t) : ch[c];
        }
        const float* g = a.gates + t * G * H + j;
        const float gi = __ldcg(g), go = __ldcg(g + H), gu = __ldcg(g + 2 * H), cown = __ldcg(a.state + t * 2 * H + H + j);
        float gf[K], cch[K];
#pragma unroll
        for (int c = 0; c < K; ++c) {
          gf[c] = __ldcg(g + (3 + c) * H);
          cch[c] = ch[c] >= 0 ? __ldcg(a.state + static_cast<size_t>(chs[c]) * 2 * H + H + j) : 0.0f;
        }
        const float mh = has_parent ? __ldcg(a.mailbox + t * 2 * H + j) : 0.0f, mc = has_parent ? __ldcg(a.mailbox + t * 2 * H + H + j) : 0.0f;
        float d_out = 0.0f;
        if (a.dz != nullptr) {
#pragma unroll
          for (int c = 0; c < kHeadDzPitch; ++c)
            if (c < a.C) d_out = fmaf(__ldg(a.dz + t * kHeadDzPitch + c), wc[c], d_out);
        } else {
          d_out = __ldg(a.dOut + t * H + j);
        }
        const float dh = d_out + mh, th = tanhf(cown), d_o = dh * th;
        const float dc = mc + (dh * go) * (1.0f - th * th);
        const float zi = (dc * gu) * gi * (1.0f - gi), zo = d_o * go * (1.0f - go), zu = (dc * gi) * (1.0f - gu * gu);
        float zfs = 0.0f;
#pragma unroll
        for (int c = 0; c < K; ++c) {
          float z = 0.0f;
          if (ch[c] >= 0) {
            z = (dc * cch[c]) * gf[c] * (1.0f - gf[c]);
            zfs += z;
            a.mailbox[static_cast<size_t>(ch[c]) * 2 * H + H + j] = dc * gf[c];
          }
          a.ZF[(t * K + c) * H + j] = z;
        }
        float* d = a.dA + t * 4 * H + j;
        d[0] = zi; d[H] = zo; d[2 * H] = zu; d[3 * H] = zfs;
        sums[0] += zi; sums[1] += zo; sums[2] += zu; sums[3] += zfs;
      }
    }
    if (!GridSync(a.barrier, ++barrier * gridDim.x, a.status)) return;
    const int tiles = (end - off + TR - 1) / TR;
    for (int tile = rg; tile < tiles; tile += a.row_groups) {
      const int t0 = off + tile * TR, rows = min(TR, end - t0);
      float ds[RPT][NPT], dq[K][RPT][NPT];
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int n = 0; n < NPT; ++n) {
          ds[r][n] = 0.0f;
#pragma unroll
          for (int c = 0; c < K; ++c) dq[c][r][n] = 0.0f;
        }
#pragma unroll
      for (int q = 0; q < G; ++q) {
        if (q % a.buffers == 0) {
          __syncthreads();   // readers of the buffers (and, at q = 0, of the sums) are done
          const int count = min(a.buffers, G - q);
          LoadRows<V>(At, p, count * TR, H, [&](int r) -> const float* {
            const int qq = q + r / TR, i = r % TR;
            if (i >= rows) return nullptr;
            const size_t t = t0 + i;
            return qq < 3 ? a.dA + t * 4 * H + qq * H : a.ZF + (t * K + qq - 3) * H;
          });
          __syncthreads();
        }
        const float* buf = At + (q % a.buffers) * TR * p;
        const float* wt = Wt + unit * pw + min(q, 3) * hk;
        if (q < 3) BwdProducts<RPT, NPT>(ds, buf, p, wt, pw, k4_begin, k4_end, lane);
        else BwdProducts<RPT, NPT>(dq[q < 3 ? 0 : q - 3], buf, p, wt, pw, k4_begin, k4_end, lane);
      }
      float* my_red = red + slice * TR * w * (1 + K);
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int n = 0; n < NPT; ++n) {
          float* x = my_red + (((lane >> 2) + r * 8) * w + unit + n * 4) * (1 + K);
          x[0] = ds[r][n];
#pragma unroll
          for (int c = 0; c < K; ++c) x[1 + c] = dq[c][r][n];
        }
      __syncthreads();
      const int prow = threadIdx.x / w, col = n0 + threadIdx.x % w;
      if (prow < rows && col < H) {
        float z[1 + K];
#pragma unroll
        for (int c = 0; c <= K; ++c) z[c] = 0.0f;
        for (int s = 0; s < slices; ++s)
#pragma unroll
          for (int c = 0; c <= K; ++c) z[c] += red[((s * TR + prow) * w + threadIdx.x % w) * (1 + K) + c];
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const int chn = __ldg(a.child + static_cast<size_t>(c) * a.n_total + t0 + prow);
          if (chn >= 0) a.mailbox[static_cast<size_t>(chn) * 2 * H + col] = z[0] + z[1 + c];
        }
      }
    }
    end = off; off = next_off;
    if (l > a.level_begin && !GridSync(a.barrier, ++barrier * gridDim.x, a.status)) return;
  }
  if (a.dB_part == nullptr) return;
  // Column sums of this CTA's rows, row lanes folded in order, into its row of dB_part.
  __syncthreads();
#pragma unroll
  for (int g = 0; g < 4; ++g) red[g * kThreads + threadIdx.x] = sums[g];
  __syncthreads();
  if (owner && threadIdx.x < kColBlock) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float acc = 0.0f;
      for (int r = 0; r < kRowLanes; ++r) acc += red[g * kThreads + r * kColBlock + threadIdx.x];
      a.dB_part[static_cast<size_t>(blockIdx.x) * 4 * H + g * H + j] += acc;
    }
  }
}

constexpr size_t kMaxSmem = 226 * 1024;

size_t ForwardSmem(int H, int K, int w) {
  const int hk = Pad4(H), tr = K <= 2 ? 32 : 16, slices = kWarps / (w / 4);
  return sizeof(float) * (static_cast<size_t>(hk) * w * 4 + static_cast<size_t>(K) * tr * Pitch(hk) + static_cast<size_t>(slices) * tr * w * (3 + K));
}
int BackwardNpt(int w) { return w >= 8 ? 2 : 1; }
size_t BackwardSmem(int H, int K, int w, int buffers) {
  const int hk = Pad4(H), tr = K <= 2 ? 32 : 16, slices = kWarps / (w / (4 * BackwardNpt(w)));
  const size_t red = std::max(static_cast<size_t>(slices) * tr * w * (1 + K), static_cast<size_t>(4) * kThreads);
  return sizeof(float) * (static_cast<size_t>(w) * Pitch(4 * hk) + static_cast<size_t>(buffers) * tr * Pitch(hk) + red);
}

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

NarrowPlan PlanNarrow(int H, int K, int rows, bool backward) {
  NarrowPlan best;
  const int tr = K <= 2 ? 32 : 16;
  const int tiles = (rows + tr - 1) / tr;
  double best_cost = 0.0;
  for (int w : {4, 8, 16}) {
    const int cols = (H + w - 1) / w;
    if (cols > SmCount()) continue;
    NarrowPlan p;
    p.w = w;
    p.col_groups = cols;
    p.row_groups = std::min(SmCount() / cols, tiles);
    p.buffers = 3 + K;
    if (backward) {
      while (p.buffers > 0 && BackwardSmem(H, K, w, p.buffers) > kMaxSmem) --p.buffers;
      if (p.buffers == 0) continue;
      p.smem = BackwardSmem(H, K, w, p.buffers);
    } else {
      p.smem = ForwardSmem(H, K, w);
      if (p.smem > kMaxSmem) continue;
    }
    // us per level: row tiles in sequence, each a gather round trip and its fused multiply-adds at about 70 % of the pipe
    const double shots = backward ? (3 + K + p.buffers - 1) / p.buffers : 1;
    const double cost = ((tiles + p.row_groups - 1) / p.row_groups) * (1.2 * shots + static_cast<double>(tr) * w * H * (3 + K) / (128.0 * 0.7 * 1900.0));
    if (best.w == 0 || cost < best_cost) { best = p; best_cost = cost; }
  }
  best.level_us = 3.0 + best_cost;
  return best;
}

int LaunchNarrowForward(const NarrowPlan& plan, NarrowForwardArgs a, int K, cudaStream_t st) {
  a.w = plan.w; a.col_groups = plan.col_groups; a.row_groups = plan.row_groups;
  const int grid = plan.col_groups * plan.row_groups;
  switch (K) {
    case 1: return ForwardK<1>(a, grid, plan.smem, st);
    case 2: return ForwardK<2>(a, grid, plan.smem, st);
    case 3: return ForwardK<3>(a, grid, plan.smem, st);
    default: return ForwardK<4>(a, grid, plan.smem, st);
  }
}

int LaunchNarrowBackward(const NarrowPlan& plan, NarrowBackwardArgs a, int K, cudaStream_t st) {
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
