// Fused child-sum Tree-GRU cell kernels (an extension: the reference has no GRU vertex function;
// the definition is the CPU oracle's, oracle/cavs_oracle.c).  Per vertex, with children h_k:
//   ht = sum_k h_k                         r_k = sigmoid((a_r + h_k U_r) + b_r)
//   z  = sigmoid((a_z + ht U_z) + b_z)     m   = sum_k r_k o h_k
//   n  = tanh((a_n + m U_n) + b_n)         h   = (1 - z) o ht + z o n
// a = x.W comes from the per-token input projection (one row per distinct token, read through
// a_row); the three recurrent products are GEMMs between these kernels.  The state row is h only.
// Same structure as the Tree-LSTM kernels (kernels/cell.cu): HBM-bound, one thread per V = 4 hidden units of one
// vertex (2 or 1 where the width is no multiple), all its loads issued before the arithmetic, grids capped at SMs x
// resident CTAs.
#include <cuda_bf16.h>

#include <cstdint>

#include "abi_common.h"
#include "kernels/gru.h"
#include "kernels/launch.h"

namespace cavs_b200 {
namespace {

constexpr int kThreads = 256;

// V consecutive values as floats: one 4 V-byte (fp32) or 2 V-byte (bf16) access.
template <int V> struct Vec { float v[V]; };
template <int V>
__device__ __forceinline__ Vec<V> Ld(const float* p) {
  Vec<V> r;
  if constexpr (V == 4) { const float4 t = *reinterpret_cast<const float4*>(p); r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w; }
  else if constexpr (V == 2) { const float2 t = *reinterpret_cast<const float2*>(p); r.v[0] = t.x; r.v[1] = t.y; }
  else r.v[0] = *p;
  return r;
}
template <int V>
__device__ __forceinline__ Vec<V> Ld(const __nv_bfloat16* p) {
  Vec<V> r;
  if constexpr (V == 4) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = b.x; r.v[3] = b.y;
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[e] = __bfloat162float(p[e]);
  }
  return r;
}
template <int V>
__device__ __forceinline__ void St(float* p, const Vec<V>& r) {
  if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(r.v[0], r.v[1]);
  else *p = r.v[0];
}
template <int V>
__device__ __forceinline__ void St(__nv_bfloat16* p, const Vec<V>& r) {
  if constexpr (V == 4) {
    __nv_bfloat162 a = __floats2bfloat162_rn(r.v[0], r.v[1]), b = __floats2bfloat162_rn(r.v[2], r.v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) p[e] = __float2bfloat16_rn(r.v[e]);
  }
}
template <int V>
__device__ __forceinline__ Vec<V> Zero() {
  Vec<V> r;
#pragma unroll
  for (int e = 0; e < V; ++e) r.v[e] = 0.0f;
  return r;
}
// The V values of a child's row, zeros for an empty slot.
template <int V>
__device__ __forceinline__ Vec<V> LdChild(const float* state, int ch, int H, int j) {
  return ch >= 0 ? Ld<V>(state + static_cast<size_t>(ch) * H + j) : Zero<V>();
}
// Sum of the children's rows, in slot order.
template <int K, int V>
__device__ __forceinline__ Vec<V> SumChildren(const float* state, const int32_t* child, size_t n_total, size_t t, int H, int j) {
  Vec<V> h[K];
#pragma unroll
  for (int c = 0; c < K; ++c) h[c] = LdChild<V>(state, __ldg(child + c * n_total + t), H, j);
#pragma unroll
  for (int c = 1; c < K; ++c)
#pragma unroll
    for (int e = 0; e < V; ++e) h[0].v[e] += h[c].v[e];
  return h[0];
}

__device__ __forceinline__ float Sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }

#define GRU_LOOP(rows, H)                                                                                                   \
  const unsigned hv = (H) / V;                                                                                              \
  const unsigned long long total = static_cast<unsigned long long>(rows) * hv;                                              \
  const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * kThreads;                                  \
  for (unsigned long long i = static_cast<unsigned long long>(blockIdx.x) * kThreads + threadIdx.x; i < total; i += stride)
// Row b of the level and first of the V hidden units.  (Row x unit counts beyond 2^32 take the 64-bit division.)
#define GRU_INDEX(b, j)                                                                                                     \
  const unsigned b = total <= 0xffffffffull ? static_cast<unsigned>(i) / hv : static_cast<unsigned>(i / hv);                \
  const int j = static_cast<int>(i - static_cast<unsigned long long>(b) * hv) * V

// r_k and m = sum_k r_k o h_k for the level's rows.  R [n_total,K,H] fp32 (saved), M [n_total,H] (GEMM operand).  Empty
// slots have no gate: nothing is read or stored for them (the backward kernels skip them the same way).
template <typename T, int K, int V>
__global__ void __launch_bounds__(kThreads)
GruGateR(float* __restrict__ R, T* __restrict__ M, const T* __restrict__ A, const T* __restrict__ PR,
         const float* __restrict__ bias, const float* __restrict__ state, const int32_t* __restrict__ child,
         const int32_t* __restrict__ a_row, int n_total, int off, int rows, int H) {
  GRU_LOOP(rows, H) {
    GRU_INDEX(b, j);
    const size_t t = static_cast<size_t>(off) + b;
    int ch[K];
#pragma unroll
    for (int c = 0; c < K; ++c) ch[c] = __ldg(child + static_cast<size_t>(c) * n_total + t);
    const Vec<V> ar = Ld<V>(A + static_cast<size_t>(a_row ? __ldg(a_row + t) : t) * 3 * H + j), br = Ld<V>(bias + j);
    Vec<V> hc[K], p[K], m = Zero<V>();
#pragma unroll
    for (int c = 0; c < K; ++c) {
      hc[c] = LdChild<V>(state, ch[c], H, j);
      p[c] = ch[c] >= 0 ? Ld<V>(PR + (static_cast<size_t>(b) * K + c) * H + j) : Zero<V>();
    }
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (ch[c] < 0) continue;
      Vec<V> r;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        r.v[e] = Sigmoid((ar.v[e] + p[c].v[e]) + br.v[e]);
        m.v[e] += r.v[e] * hc[c].v[e];
      }
      St<V>(R + (t * K + c) * H + j, r);
    }
    St<V>(M + t * H + j, m);
  }
}

// z, n and the new state.  ZN [n_total,2H] fp32 (saved).  kLeaf: no children (pz = pn = 0, ht = 0).
template <typename T, int K, int V, bool kLeaf>
__global__ void __launch_bounds__(kThreads)
GruOut(float* __restrict__ state, float* __restrict__ ZN, const T* __restrict__ A, const T* __restrict__ PZ,
       const T* __restrict__ PN, const float* __restrict__ bias, const int32_t* __restrict__ child,
       const int32_t* __restrict__ a_row, int n_total, int off, int rows, int H) {
  GRU_LOOP(rows, H) {
    GRU_INDEX(b, j);
    const size_t t = static_cast<size_t>(off) + b;
    const T* a = A + static_cast<size_t>(a_row ? __ldg(a_row + t) : t) * 3 * H + j;
    const Vec<V> az = Ld<V>(a + H), an = Ld<V>(a + 2 * H), bz = Ld<V>(bias + H + j), bn = Ld<V>(bias + 2 * H + j);
    Vec<V> ht = Zero<V>(), pz = Zero<V>(), pn = Zero<V>();
    if (!kLeaf) {
      pz = Ld<V>(PZ + static_cast<size_t>(b) * H + j);
      pn = Ld<V>(PN + static_cast<size_t>(b) * H + j);
      ht = SumChildren<K, V>(state, child, n_total, t, H, j);
    }
    Vec<V> z, n, h;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      z.v[e] = Sigmoid((az.v[e] + pz.v[e]) + bz.v[e]);
      n.v[e] = tanhf((an.v[e] + pn.v[e]) + bn.v[e]);
      h.v[e] = (1.0f - z.v[e]) * ht.v[e] + z.v[e] * n.v[e];
    }
    St<V>(ZN + t * 2 * H + j, z);
    St<V>(ZN + t * 2 * H + H + j, n);
    St<V>(state + t * H + j, h);
  }
}

// First backward stage: dh = dOut + parent's message; writes the z / n pre-activation gradients into
// dA's blocks 1, 2 and d(ht) into the level-local dHt; leaves also zero dA's r block.
template <typename T, int K, int V, bool kLeaf>
__global__ void __launch_bounds__(kThreads)
GruBwdA(T* __restrict__ dA, float* __restrict__ dHt, const float* __restrict__ mailbox, const float* __restrict__ dOut,
        const float* __restrict__ ZN, const float* __restrict__ state, const int32_t* __restrict__ child,
        const int32_t* __restrict__ parent, int n_total, int off, int rows, int H) {
  GRU_LOOP(rows, H) {
    GRU_INDEX(b, j);
    const size_t t = static_cast<size_t>(off) + b;
    const bool has_parent = __ldg(parent + t) >= 0;
    Vec<V> dh = Ld<V>(dOut + t * H + j);
    const Vec<V> z = Ld<V>(ZN + t * 2 * H + j), n = Ld<V>(ZN + t * 2 * H + H + j);
    const Vec<V> mail = has_parent ? Ld<V>(mailbox + t * H + j) : Zero<V>();
    Vec<V> ht = Zero<V>(), zz, zn, dht;
    if (!kLeaf) ht = SumChildren<K, V>(state, child, n_total, t, H, j);
#pragma unroll
    for (int e = 0; e < V; ++e) {
      dh.v[e] += mail.v[e];
      zz.v[e] = (dh.v[e] * (n.v[e] - ht.v[e])) * z.v[e] * (1.0f - z.v[e]);
      zn.v[e] = (dh.v[e] * z.v[e]) * (1.0f - n.v[e] * n.v[e]);
      dht.v[e] = dh.v[e] * (1.0f - z.v[e]);
    }
    St<V>(dA + t * 3 * H + H + j, zz);
    St<V>(dA + t * 3 * H + 2 * H + j, zn);
    if (kLeaf) St<V>(dA + t * 3 * H + j, Zero<V>());
    else St<V>(dHt + static_cast<size_t>(b) * H + j, dht);
  }
}

// Second stage: zr_k = (dm o h_k) r_k (1 - r_k) -> ZR [n_total,K,H] (GEMM operand), dA block 0 = sum_k zr_k.
template <typename T, int K, int V>
__global__ void __launch_bounds__(kThreads)
GruBwdB1(T* __restrict__ dA, T* __restrict__ ZR, const float* __restrict__ dm, const float* __restrict__ R,
         const float* __restrict__ state, const int32_t* __restrict__ child, int n_total, int off, int rows, int H) {
  GRU_LOOP(rows, H) {
    GRU_INDEX(b, j);
    const size_t t = static_cast<size_t>(off) + b;
    int ch[K];
#pragma unroll
    for (int c = 0; c < K; ++c) ch[c] = __ldg(child + static_cast<size_t>(c) * n_total + t);
    const Vec<V> d = Ld<V>(dm + static_cast<size_t>(b) * H + j);
    Vec<V> hc[K], r[K], acc = Zero<V>();
#pragma unroll
    for (int c = 0; c < K; ++c) {
      hc[c] = LdChild<V>(state, ch[c], H, j);
      r[c] = ch[c] >= 0 ? Ld<V>(R + (t * K + c) * H + j) : Zero<V>();
    }
#pragma unroll
    for (int c = 0; c < K; ++c) {
      Vec<V> zr;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        zr.v[e] = ch[c] >= 0 ? (d.v[e] * hc[c].v[e]) * r[c].v[e] * (1.0f - r[c].v[e]) : 0.0f;
        acc.v[e] += zr.v[e];
      }
      St<V>(ZR + (t * K + c) * H + j, zr);
    }
    St<V>(dA + t * 3 * H + j, acc);
  }
}

// Third stage: mailbox[child_k] = ((d(ht) + dsz) + dm o r_k) + dqr_k.
template <int K, int V>
__global__ void __launch_bounds__(kThreads)
GruBwdB2(float* __restrict__ mailbox, const float* __restrict__ dHt, const float* __restrict__ dsz,
         const float* __restrict__ dm, const float* __restrict__ dqr, const float* __restrict__ R,
         const int32_t* __restrict__ child, int n_total, int off, int rows, int H) {
  GRU_LOOP(rows, H) {
    GRU_INDEX(b, j);
    const size_t t = static_cast<size_t>(off) + b, row = static_cast<size_t>(b) * H + j;
    int ch[K];
#pragma unroll
    for (int c = 0; c < K; ++c) ch[c] = __ldg(child + static_cast<size_t>(c) * n_total + t);
    const Vec<V> x = Ld<V>(dHt + row), y = Ld<V>(dsz + row), d = Ld<V>(dm + row);
    Vec<V> r[K], q[K];
#pragma unroll
    for (int c = 0; c < K; ++c)
      if (ch[c] >= 0) {
        r[c] = Ld<V>(R + (t * K + c) * H + j);
        q[c] = Ld<V>(dqr + (static_cast<size_t>(b) * K + c) * H + j);
      }
#pragma unroll
    for (int c = 0; c < K; ++c)
      if (ch[c] >= 0) {
        Vec<V> out;
#pragma unroll
        for (int e = 0; e < V; ++e) out.v[e] = ((x.v[e] + y.v[e]) + d.v[e] * r[c].v[e]) + q[c].v[e];
        St<V>(mailbox + static_cast<size_t>(ch[c]) * H + j, out);
      }
  }
}

#define DISPATCH_V(V_, ...)                                   \
  do {                                                        \
    switch (V_) {                                               \
      case 4: { constexpr int V = 4; __VA_ARGS__; break; }    \
      case 2: { constexpr int V = 2; __VA_ARGS__; break; }    \
      default: { constexpr int V = 1; __VA_ARGS__; break; }   \
    }                                                         \
  } while (0)
#define DISPATCH_K(K_, V_, ...)                                                \
  do {                                                                         \
    switch (K_) {                                                              \
      case 1: { constexpr int K = 1; DISPATCH_V(V_, __VA_ARGS__); break; }     \
      case 2: { constexpr int K = 2; DISPATCH_V(V_, __VA_ARGS__); break; }     \
      case 3: { constexpr int K = 3; DISPATCH_V(V_, __VA_ARGS__); break; }     \
      default: { constexpr int K = 4; DISPATCH_V(V_, __VA_ARGS__); break; }    \
    }                                                                          \
  } while (0)

int Check(const char* name, int rows, int H, int K) {
  CAVS_REQUIRE(rows >= 0 && H > 0 && K >= 1 && K <= 4, CAVS_ERR_BAD_ARG, std::string(name) + ": bad shape");
  return CAVS_OK;
}

}  // namespace

using bf = __nv_bfloat16;

int LaunchGruGateR(float* R, void* M, bool bf16, const void* A, const void* PR, const float* bias, const float* state,
                   const int32_t* child, const int32_t* a_row, int n_total, int off, int rows, int H, int K, cudaStream_t st) {
  if (int rc = Check("gru_gate_r", rows, H, K)) return rc;
  if (rows == 0) return CAVS_OK;
  const int vec = VecWidth(H, bias), grid = GridForElems(static_cast<size_t>(rows) * (H / vec), kThreads);
  DISPATCH_K(K, vec, {
    if (bf16) GruGateR<bf, K, V><<<grid, kThreads, 0, st>>>(R, static_cast<bf*>(M), static_cast<const bf*>(A), static_cast<const bf*>(PR), bias, state, child, a_row, n_total, off, rows, H);
    else GruGateR<float, K, V><<<grid, kThreads, 0, st>>>(R, static_cast<float*>(M), static_cast<const float*>(A), static_cast<const float*>(PR), bias, state, child, a_row, n_total, off, rows, H);
  });
  CAVS_LAUNCH_CHECK("gru_gate_r");
  return CAVS_OK;
}

int LaunchGruOut(float* state, float* ZN, bool bf16, const void* A, const void* PZ, const void* PN, const float* bias,
                 const int32_t* child, const int32_t* a_row, int n_total, int off, int rows, int H, int K, bool leaf,
                 cudaStream_t st) {
  if (int rc = Check("gru_out", rows, H, K)) return rc;
  if (rows == 0) return CAVS_OK;
  const int vec = VecWidth(H, bias), grid = GridForElems(static_cast<size_t>(rows) * (H / vec), kThreads);
  DISPATCH_K(K, vec, {
    if (bf16) {
      auto a = static_cast<const bf*>(A); auto pz = static_cast<const bf*>(PZ); auto pn = static_cast<const bf*>(PN);
      if (leaf) GruOut<bf, K, V, true><<<grid, kThreads, 0, st>>>(state, ZN, a, pz, pn, bias, child, a_row, n_total, off, rows, H);
      else GruOut<bf, K, V, false><<<grid, kThreads, 0, st>>>(state, ZN, a, pz, pn, bias, child, a_row, n_total, off, rows, H);
    } else {
      auto a = static_cast<const float*>(A); auto pz = static_cast<const float*>(PZ); auto pn = static_cast<const float*>(PN);
      if (leaf) GruOut<float, K, V, true><<<grid, kThreads, 0, st>>>(state, ZN, a, pz, pn, bias, child, a_row, n_total, off, rows, H);
      else GruOut<float, K, V, false><<<grid, kThreads, 0, st>>>(state, ZN, a, pz, pn, bias, child, a_row, n_total, off, rows, H);
    }
  });
  CAVS_LAUNCH_CHECK("gru_out");
  return CAVS_OK;
}

int LaunchGruBwdA(void* dA, float* dHt, bool bf16, const float* mailbox, const float* dOut, const float* ZN, const float* state,
                  const int32_t* child, const int32_t* parent, int n_total, int off, int rows, int H, int K, bool leaf,
                  cudaStream_t st) {
  if (int rc = Check("gru_bwd_a", rows, H, K)) return rc;
  if (rows == 0) return CAVS_OK;
  const int vec = VecWidth(H), grid = GridForElems(static_cast<size_t>(rows) * (H / vec), kThreads);
  DISPATCH_K(K, vec, {
    if (bf16) {
      if (leaf) GruBwdA<bf, K, V, true><<<grid, kThreads, 0, st>>>(static_cast<bf*>(dA), dHt, mailbox, dOut, ZN, state, child, parent, n_total, off, rows, H);
      else GruBwdA<bf, K, V, false><<<grid, kThreads, 0, st>>>(static_cast<bf*>(dA), dHt, mailbox, dOut, ZN, state, child, parent, n_total, off, rows, H);
    } else {
      if (leaf) GruBwdA<float, K, V, true><<<grid, kThreads, 0, st>>>(static_cast<float*>(dA), dHt, mailbox, dOut, ZN, state, child, parent, n_total, off, rows, H);
      else GruBwdA<float, K, V, false><<<grid, kThreads, 0, st>>>(static_cast<float*>(dA), dHt, mailbox, dOut, ZN, state, child, parent, n_total, off, rows, H);
    }
  });
  CAVS_LAUNCH_CHECK("gru_bwd_a");
  return CAVS_OK;
}

int LaunchGruBwdB1(void* dA, void* ZR, bool bf16, const float* dm, const float* R, const float* state, const int32_t* child,
                   int n_total, int off, int rows, int H, int K, cudaStream_t st) {
  if (int rc = Check("gru_bwd_b1", rows, H, K)) return rc;
  if (rows == 0) return CAVS_OK;
  const int vec = VecWidth(H), grid = GridForElems(static_cast<size_t>(rows) * (H / vec), kThreads);
  DISPATCH_K(K, vec, {
    if (bf16) GruBwdB1<bf, K, V><<<grid, kThreads, 0, st>>>(static_cast<bf*>(dA), static_cast<bf*>(ZR), dm, R, state, child, n_total, off, rows, H);
    else GruBwdB1<float, K, V><<<grid, kThreads, 0, st>>>(static_cast<float*>(dA), static_cast<float*>(ZR), dm, R, state, child, n_total, off, rows, H);
  });
  CAVS_LAUNCH_CHECK("gru_bwd_b1");
  return CAVS_OK;
}

int LaunchGruBwdB2(float* mailbox, const float* dHt, const float* dsz, const float* dm, const float* dqr, const float* R,
                   const int32_t* child, int n_total, int off, int rows, int H, int K, cudaStream_t st) {
  if (int rc = Check("gru_bwd_b2", rows, H, K)) return rc;
  if (rows == 0) return CAVS_OK;
  const int vec = VecWidth(H), grid = GridForElems(static_cast<size_t>(rows) * (H / vec), kThreads);
  DISPATCH_K(K, vec, { GruBwdB2<K, V><<<grid, kThreads, 0, st>>>(mailbox, dHt, dsz, dm, dqr, R, child, n_total, off, rows, H); });
  CAVS_LAUNCH_CHECK("gru_bwd_b2");
  return CAVS_OK;
}

}  // namespace cavs_b200
