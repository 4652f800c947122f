// The narrow levels of the bf16 Tree-LSTM in one launch per direction (see narrow_f32.cu for the scheme): a persistent
// grid walks the levels with a bounded grid barrier between them, each CTA keeps its eight hidden units' slice of the
// recurrent weights in shared memory.  One child slot, H = 512, 49 rows on average: 15.6 -> 6.1 us per level forward,
// 23.6 -> 9 us backward; two stacked layers of 60 levels 3.80 -> 2.50 ms per step.
//
// Level by level a narrow level costs 16 us forward (child gather, both gate products in one launch, cell) and 23 us
// backward (cell gradient, two products) at H = 512, of which the tensor cores work a fraction of a microsecond.
// The products here are mma.sync m16n8k16 on fragments from shared memory: one n8 tile is exactly the CTA's eight
// units of a gate, the k range is cut over the sixteen warps.  tcgen05 would need 128-row tiles, of which a level of 16
// to 100 rows fills a part, and a TMEM round trip per level; wide levels keep the tcgen05 kernels.
#include <algorithm>

#include "kernels/narrow.cuh"

namespace cavs_b200 {
namespace {

using namespace narrow;
using bf16 = __nv_bfloat16;

constexpr int kUnits = 8;                                            // hidden units per CTA: one n8 tile per gate
template <int K> constexpr int TileRows() { return K == 1 ? 32 : 16; }
// Row pitch in elements: a multiple of 64 plus 8, so that the eight rows of an ldmatrix start in different bank groups.
__host__ __device__ inline int Pitch(int H) { return ((H + 63) & ~63) + 8; }

__device__ __forceinline__ uint32_t SmemAddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void LdMatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void LdMatrix2(uint32_t (&r)[2], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void Mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint2 Pack4(const float4& v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}

// ---- forward ----
template <int K>
__global__ void __launch_bounds__(kThreads, 1) NarrowForwardBf16(const NarrowForwardArgs a) {
  constexpr int TR = TileRows<K>(), MT = TR / 16, G = 3 + K, NV = K == 1 ? 1 : K + 1;   // NV: h of each child, then their sum
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ int s_child[K][TR];
  const int H = a.H, pk = Pitch(H), steps = (H + 15) / 16;
  bf16* Wb = reinterpret_cast<bf16*>(smem_raw);        // [4 gates i, o, u, f][8 units][pk]
  bf16* At = Wb + 4 * kUnits * pk;                     // [NV][TR][pk]
  // [warps][G][TR][8]: a fragment's float2 stores and the sums' reads fall into all banks
  float* red = reinterpret_cast<float*>(At + NV * TR * pk);
  const int cg = blockIdx.x % a.col_groups, rg = blockIdx.x / a.col_groups, j0 = cg * kUnits;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = (steps + kWarps - 1) / kWarps, step_begin = min(steps, warp * per), step_end = min(steps, step_begin + per);
  for (int i = threadIdx.x; i < (4 * kUnits + NV * TR) * pk / 8; i += kThreads) reinterpret_cast<uint4*>(Wb)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * H; i += kThreads) {   // eight units of one gate at one k: 16 bytes
    const int g = i & 3, k = i >> 2;
    const bf16* u = g < 3 ? static_cast<const bf16*>(a.U_iou) + static_cast<size_t>(k) * 3 * H + g * H + j0
                          : static_cast<const bf16*>(a.U_f) + static_cast<size_t>(k) * H + j0;
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(u));
    const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
    for (int n = 0; n < kUnits; ++n) Wb[(g * kUnits + n) * pk + k] = e[n];
  }
  const int prow = threadIdx.x / kUnits, pu = threadIdx.x % kUnits, pj = j0 + pu;
  const bool pair = prow < TR;
  float bi = 0.f, bf = 0.f, bu = 0.f, bo = 0.f;
  if (pair) { bi = a.bias[pj]; bf = a.bias[H + pj]; bu = a.bias[2 * H + pj]; bo = a.bias[3 * H + pj]; }

  int off = __ldg(a.level_off + a.level_begin), end = __ldg(a.level_off + a.level_begin + 1);
  unsigned barrier = 0;
  int child = -1;
  float in[4] = {};
  auto prefetch = [&](int off_, int end_, int tile) {   // what a tile needs beside the previous level's states
    child = -1;
    const int t = off_ + tile * TR + static_cast<int>(threadIdx.x) % TR;
    if (threadIdx.x < K * TR && t < end_) child = __ldg(a.child + static_cast<size_t>(threadIdx.x / TR) * a.n_total + t);
    const int tp = off_ + tile * TR + prow;
    if (pair && tp < end_) {
      const bf16* x = static_cast<const bf16*>(a.A) + static_cast<size_t>(a.a_row ? __ldg(a.a_row + tp) : tp) * 4 * H + pj;
#pragma unroll
      for (int g = 0; g < 4; ++g) in[g] = __bfloat162float(x[g * H]);
    }
  };
  prefetch(off, end, rg);
  const int b_row = lane & 7, b_col = ((lane >> 3) & 1) * 8, b_gate = lane >> 4;   // ldmatrix: two gates, two k halves
  const uint32_t b_addr = SmemAddr(Wb + (b_gate * kUnits + b_row) * pk + b_col), b_pair = 2 * kUnits * pk * 2;
  const uint32_t a_addr = SmemAddr(At + (lane & 15) * pk + (lane >> 4) * 8);
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
      for (int c = 0; c < K; ++c) {
        const int ch = pair && prow < rows ? s_child[c][prow] : -1;
        c_in[c] = ch >= 0 ? __ldcg(a.state + static_cast<size_t>(ch) * 2 * H + H + pj) : 0.0f;
      }
      // children's h rows (fp32, L1 bypassed) -> bf16 rows and their sum, four rows in flight per thread
      for (int r0 = threadIdx.x >> 7; r0 < rows; r0 += 16)
        for (int j = (threadIdx.x & 127) * 4; j < H; j += 512) {
          float4 h[4][K];
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int c = 0; c < K; ++c) {
              const int r = r0 + u * 4, ch = r < rows ? s_child[c][r] : -1;
              h[u][c] = ch >= 0 ? __ldcg(reinterpret_cast<const float4*>(a.state + static_cast<size_t>(ch) * 2 * H + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int r = r0 + u * 4;
            if (r >= rows) break;
            float4 s = h[u][0];
#pragma unroll
            for (int c = 0; c < K; ++c) {
              *reinterpret_cast<uint2*>(At + (c * TR + r) * pk + j) = Pack4(h[u][c]);
              if (c > 0) { s.x += h[u][c].x; s.y += h[u][c].y; s.z += h[u][c].z; s.w += h[u][c].w; }
            }
            if (K > 1) *reinterpret_cast<uint2*>(At + (K * TR + r) * pk + j) = Pack4(s);
          }
        }
      __syncthreads();
      float acc[MT][G][4];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[m][g][e] = 0.0f;
      for (int st = step_begin; st < step_end; ++st) {
        uint32_t b01[4], b23[4];   // gates i, o and u, f
        LdMatrix4(b01, b_addr + st * 32);
        LdMatrix4(b23, b_addr + b_pair + st * 32);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          if (m * 16 >= rows) break;
          uint32_t s[4];
          LdMatrix4(s, a_addr + ((NV - 1) * TR + m * 16) * pk * 2 + st * 32);
          Mma(acc[m][0], s, b01[0], b01[1]);
          Mma(acc[m][1], s, b01[2], b01[3]);
          Mma(acc[m][2], s, b23[0], b23[1]);
          if (K == 1) {
            Mma(acc[m][3], s, b23[2], b23[3]);
          } else {
#pragma unroll
            for (int c = 0; c < K; ++c) {
              uint32_t h[4];
              LdMatrix4(h, a_addr + (c * TR + m * 16) * pk * 2 + st * 32);
              Mma(acc[m][3 + c], h, b23[2], b23[3]);
            }
          }
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int e = 0; e < 4; e += 2)
            *reinterpret_cast<float2*>(red + ((warp * G + g) * TR + m * 16 + (lane >> 2) + e * 4) * kUnits + (lane & 3) * 2) =
                make_float2(acc[m][g][e], acc[m][g][e + 1]);
      __syncthreads();
      if (pair && prow < rows) {
        float z[G];
#pragma unroll
        for (int g = 0; g < G; ++g) z[g] = 0.0f;
#pragma unroll
        for (int s = 0; s < kWarps; ++s)
#pragma unroll
          for (int g = 0; g < G; ++g) z[g] += red[(s * G + g) * TR * kUnits + threadIdx.x];
        const size_t t = t0 + prow;
        const float gi = Sigmoid<true>((in[0] + z[0]) + bi), go = Sigmoid<true>((in[1] + z[1]) + bo), gu = Tanh<true>((in[2] + z[2]) + bu);
        float cc = gi * gu;
        __half* g = static_cast<__half*>(a.gates) + t * a.pitch3 + pj;
        __half* f = static_cast<__half*>(a.gates_f) + t * a.pitch_f + pj;
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const float gf = Sigmoid<true>((in[3] + z[3 + c]) + bf);
          cc = cc + gf * c_in[c];
          StoreAs(f + c * H, gf);
          static_cast<bf16*>(a.HK)[(t * K + c) * H + pj] = At[(c * TR + prow) * pk + pj];
        }
        static_cast<bf16*>(a.S)[t * H + pj] = At[((NV - 1) * TR + prow) * pk + pj];
        StoreAs(g, gi); StoreAs(g + H, go); StoreAs(g + 2 * H, gu);
        a.state[t * 2 * H + pj] = go * Tanh<true>(cc);
        a.state[t * 2 * H + H + pj] = cc;
      }
    }
    off = end; end = next_end;
    if (l + 1 < a.level_end) {
      GridArrive(a.barrier);
      prefetch(off, end, rg);
      if (!GridWait(a.barrier, ++barrier * gridDim.x + a.withhold, a.status)) return;
    }
  }
}

// ---- backward ----
template <int K>
__global__ void __launch_bounds__(kThreads, 1) NarrowBackwardBf16(const NarrowBackwardArgs a) {
  constexpr int TR = TileRows<K>(), MT = TR / 16, G = 3 + K;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int H = a.H, pk = Pitch(H), steps = (H + 15) / 16;
  bf16* Wb = reinterpret_cast<bf16*>(smem_raw);        // [4 blocks i, o, u, f][8 rows n of U][pk]
  bf16* At = Wb + 4 * kUnits * pk;                     // [buffers][TR][pk]
  float* red = reinterpret_cast<float*>(At + a.buffers * TR * pk);   // [warps][1 + K][TR][8]
  const int cg = blockIdx.x % a.col_groups, rg = blockIdx.x / a.col_groups, n0 = cg * kUnits;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = (steps + kWarps - 1) / kWarps, step_begin = min(steps, warp * per), step_end = min(steps, step_begin + per);
  for (int i = threadIdx.x; i < (4 * kUnits + a.buffers * TR) * pk / 8; i += kThreads) reinterpret_cast<uint4*>(Wb)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * kUnits * (H / 8); i += kThreads) {
    const int row = i / (H / 8), k = (i - row * (H / 8)) * 8, q = row / kUnits, n = n0 + row % kUnits;
    const bf16* u = q < 3 ? static_cast<const bf16*>(a.U_iou) + static_cast<size_t>(n) * 3 * H + q * H + k
                          : static_cast<const bf16*>(a.U_f) + static_cast<size_t>(n) * H + k;
    *reinterpret_cast<uint4*>(Wb + row * pk + k) = __ldg(reinterpret_cast<const uint4*>(u));
  }
  GateGradients<K, __half, bf16> gg(a);
  __shared__ uint64_t s_full[G];
  BulkRows<G> ring;
  ring.Init(s_full, 1);
  __syncthreads();
  const uint32_t b_addr = SmemAddr(Wb + (lane & 7) * pk + ((lane >> 3) & 1) * 8);
  const uint32_t a_addr = SmemAddr(At + (lane & 15) * pk + (lane >> 4) * 8);
  const int prow = threadIdx.x / kUnits, pu = threadIdx.x % kUnits, col = n0 + pu;

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
      const bool pair = prow < rows;
      int chn[K];
#pragma unroll
      for (int c = 0; c < K; ++c) chn[c] = pair ? __ldg(a.child + static_cast<size_t>(c) * a.n_total + t0 + prow) : -1;
      // vectors zi, zo, zu, zf_0.. through a ring of buffers, one warp's copies each; rows past the level's end keep what the
      // buffer held
      auto load = [&](int q) {
        if (warp != q) return;
        const size_t t = t0 + lane;
        const bf16* s = q < 3 ? static_cast<const bf16*>(a.dA) + t * 4 * H + q * H : static_cast<const bf16*>(a.ZF) + (t * K + q - 3) * H;
        ring.Copy(q % a.buffers, SmemAddr(At + (q % a.buffers) * TR * pk), pk * 2, lane < rows ? s : nullptr, H * 2);
      };
      float ds[MT][4], dq[K][MT][4];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          ds[m][e] = 0.0f;
#pragma unroll
          for (int c = 0; c < K; ++c) dq[c][m][e] = 0.0f;
        }
      __syncthreads();   // the previous tile's readers are done
      const int ahead = min(a.buffers, G);
      for (int q = 0; q < ahead; ++q) load(q);
#pragma unroll
      for (int q = 0; q < G; ++q) {
        ring.Wait(q % a.buffers, a.status);
        for (int st = step_begin; st < step_end; ++st) {
          uint32_t b[2];
          LdMatrix2(b, b_addr + min(q, 3) * kUnits * pk * 2 + st * 32);
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            if (m * 16 >= rows) break;
            uint32_t x[4];
            LdMatrix4(x, a_addr + ((q % a.buffers) * TR + m * 16) * pk * 2 + st * 32);
            if (q < 3) Mma(ds[m], x, b[0], b[1]);
            else Mma(dq[q < 3 ? 0 : q - 3][m], x, b[0], b[1]);
          }
        }
        if (q + a.buffers < G) {
          __syncthreads();
          load(q + a.buffers);
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          float* x = red + (warp * (1 + K) * TR + m * 16 + (lane >> 2) + e * 4) * kUnits + (lane & 3) * 2;
          *reinterpret_cast<float2*>(x) = make_float2(ds[m][e], ds[m][e + 1]);
#pragma unroll
          for (int c = 0; c < K; ++c) *reinterpret_cast<float2*>(x + (1 + c) * TR * kUnits) = make_float2(dq[c][m][e], dq[c][m][e + 1]);
        }
      __syncthreads();
      if (pair) {
        float z[1 + K];
#pragma unroll
        for (int c = 0; c <= K; ++c) z[c] = 0.0f;
#pragma unroll
        for (int s = 0; s < kWarps; ++s)
#pragma unroll
          for (int c = 0; c <= K; ++c) z[c] += red[(s * (1 + K) + c) * TR * kUnits + threadIdx.x];
#pragma unroll
        for (int c = 0; c < K; ++c)
          if (chn[c] >= 0) a.mailbox[static_cast<size_t>(chn[c]) * 2 * H + col] = z[0] + z[1 + c];
      }
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

}  // namespace

NarrowPlan PlanNarrowBf16(int H, int K, int rows, bool backward) {
  NarrowPlan p;
  const int tr = K == 1 ? 32 : 16, cols = H / kUnits, tiles = (rows + tr - 1) / tr;
  if (H % kUnits != 0 || cols > SmCount()) return p;
  const size_t pk = Pitch(H), weights = 4 * kUnits * pk * 2, tile = tr * pk * 2;
  const size_t red = sizeof(float) * std::max<size_t>(static_cast<size_t>(kWarps) * tr * kUnits * (backward ? 1 + K : 3 + K), 4 * kThreads);
  p.buffers = backward ? 3 + K : (K == 1 ? 1 : K + 1);
  while (backward && p.buffers > 1 && weights + p.buffers * tile + red > kMaxSmem) --p.buffers;
  p.smem = weights + p.buffers * tile + red;
  if (p.smem > kMaxSmem) return NarrowPlan();
  p.w = kUnits;
  p.col_groups = cols;
  // us: barriers and dependent round trips, a tile's own round trips, and the rows every CTA pulls out of L2.  Backward
  // with one row group has one barrier per level instead of two, but every CTA takes every row.
  for (int groups : {1, std::min(SmCount() / cols, tiles)}) {
    const double mine = (tiles + groups - 1) / groups;
    const double bytes = static_cast<double>(cols) * rows * H * (backward ? 2.0 * (3 + K) : 4.0 * K);
    const double us = (backward ? (groups > 1 ? 7.0 : 4.5) : 3.5) + (backward ? 2.5 : 1.5) * mine + std::max(bytes / 5e6, bytes / cols / groups / 0.1e6);
    if (p.row_groups == 0 || us < p.level_us) { p.row_groups = groups; p.level_us = us; }
  }
  return p;
}

int LaunchNarrowForwardBf16(const NarrowPlan& plan, NarrowForwardArgs a, int K, cudaStream_t st) {
  a.w = plan.w; a.col_groups = plan.col_groups; a.row_groups = plan.row_groups; a.buffers = plan.buffers;
  const int grid = plan.col_groups * plan.row_groups;
  switch (K) {
    case 1: return LaunchCooperative<NarrowForwardBf16<1>>(a, grid, plan.smem, st);
    case 2: return LaunchCooperative<NarrowForwardBf16<2>>(a, grid, plan.smem, st);
    case 3: return LaunchCooperative<NarrowForwardBf16<3>>(a, grid, plan.smem, st);
    default: return LaunchCooperative<NarrowForwardBf16<4>>(a, grid, plan.smem, st);
  }
}

int LaunchNarrowBackwardBf16(const NarrowPlan& plan, NarrowBackwardArgs a, int K, cudaStream_t st) {
  a.w = plan.w; a.col_groups = plan.col_groups; a.row_groups = plan.row_groups; a.buffers = plan.buffers;
  const int grid = plan.col_groups * plan.row_groups;
  switch (K) {
    case 1: return LaunchCooperative<NarrowBackwardBf16<1>>(a, grid, plan.smem, st);
    case 2: return LaunchCooperative<NarrowBackwardBf16<2>>(a, grid, plan.smem, st);
    case 3: return LaunchCooperative<NarrowBackwardBf16<3>>(a, grid, plan.smem, st);
    default: return LaunchCooperative<NarrowBackwardBf16<4>>(a, grid, plan.smem, st);
  }
}

}  // namespace cavs_b200
