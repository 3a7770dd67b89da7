// Memory-bound MoE ops that have no counterpart in the reference (it is a pure communication
// library): router top-k + softmax + tokens-per-expert histogram and its backward, the SwiGLU
// backward (the forward is fused into the gate/up GEMM epilogue), the decoder's cross-entropy, and the
// fused SGD update of bf16 weights from fp32 grads.  All are bandwidth kernels: 16-byte vector accesses, one pass.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>

#include "host/ctx.h"
#include "host/errors.h"

namespace mep {

// ---- router: top-k over (logits + bias), softmax over the selected unbiased logits ------------
// One warp per token.  The biased logits are turned into order-preserving unsigned keys and, up to
// 32 * ROUTER_VPL experts, stay in registers; a selection round is then ROUTER_VPL compares, one
// warp-wide redux for the largest key and one for its smallest expert index.  (With the keys in
// shared memory and ten shuffles a round the kernel was bound by that chain: 18 us for 4096 tokens
// x 32 experts, top-8.)  A NaN gets the lowest key of all: it is chosen only when nothing else is
// left, and no input makes an index leave [0, E).  Selections are counted per block in shared memory:
// one global atomic per selection made the popular experts' counters the limit (15 us of 18).
constexpr int ROUTER_WARPS = 8;
constexpr int ROUTER_VPL = 8;                 // keys per lane kept in registers

__device__ __forceinline__ uint32_t router_key(float x) {
  const uint32_t b = __float_as_uint(x);
  if ((b & 0x7FFFFFFFu) > 0x7F800000u) return 1u;                 // NaN; 0 marks "already selected"
  if (b == 0x80000000u) return b;                                 // -0 ties with +0
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);              // (-inf maps to 0x007FFFFF)
}

template <bool REGS>
__global__ void __launch_bounds__(ROUTER_WARPS * 32)
ep_router_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int S, int E,
                      int K, int32_t* __restrict__ topk, float* __restrict__ weights,
                      int32_t* __restrict__ tpe) {
  extern __shared__ uint32_t s_hist[];   // [E] selections, then [warps][E] keys unless they fit in registers
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (int)(blockDim.x >> 5);
  uint32_t* sk = REGS ? nullptr : s_hist + E + (size_t)warp * E;
  for (int e = threadIdx.x; e < E; e += (int)blockDim.x) s_hist[e] = 0u;
  __syncthreads();
  for (int s = blockIdx.x * nwarps + warp; s < S; s += gridDim.x * nwarps) {
    const float* row = logits + (size_t)s * E;
    uint32_t key[ROUTER_VPL];
    if constexpr (REGS) {
#pragma unroll
      for (int i = 0; i < ROUTER_VPL; ++i) {
        const int e = i * 32 + lane;
        key[i] = e < E ? router_key(row[e] + (bias ? bias[e] : 0.f)) : 0u;
      }
    } else {
      for (int e = lane; e < E; e += 32) sk[e] = router_key(row[e] + (bias ? bias[e] : 0.f));
      __syncwarp();
    }
    int sel_idx = 0;         // lane k keeps the k-th selected expert
    for (int k = 0; k < K; ++k) {
      uint32_t best = 0u;
      int at = E - 1;        // smallest index of this lane's largest key
      if constexpr (REGS) {
#pragma unroll
        for (int i = 0; i < ROUTER_VPL; ++i)
          if (key[i] > best) { best = key[i]; at = i * 32 + lane; }
      } else {
        for (int e = lane; e < E; e += 32) {
          const uint32_t x = sk[e];
          if (x > best) { best = x; at = e; }
        }
      }
      const uint32_t top = __reduce_max_sync(0xffffffffu, best);
      const int idx = (int)__reduce_min_sync(0xffffffffu, best == top ? (uint32_t)at : (uint32_t)(E - 1));
      if (lane == k) sel_idx = idx;
      if constexpr (REGS) {
#pragma unroll
        for (int i = 0; i < ROUTER_VPL; ++i)
          if (i * 32 + lane == idx) key[i] = 0u;
      } else {
        if (lane == 0) sk[idx] = 0u;
        __syncwarp();
      }
    }
    // softmax over the K selected logits (lanes 0..K-1)
    const float sel_logit = lane < K ? row[sel_idx] : -FLT_MAX;
    float m = sel_logit;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float ex = lane < K ? __expf(sel_logit - m) : 0.f;
    float sum = ex;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane < K) {
      topk[(size_t)s * K + lane] = sel_idx;
      weights[(size_t)s * K + lane] = ex / sum;
      atomicAdd(&s_hist[sel_idx], 1u);
    }
    if constexpr (!REGS) __syncwarp();
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += (int)blockDim.x)
    if (s_hist[e] != 0u) atomicAdd(&tpe[e], (int)s_hist[e]);
}

// d logits = softmax backward scattered to the selected experts (zero elsewhere), bf16 so that
// it can feed the tensor-core GEMMs of the router's weight and input gradients.
__global__ void ep_router_topk_bwd_kernel(const float* __restrict__ weights, const float* __restrict__ dweights,
                                          const int32_t* __restrict__ topk, int S, int E, int K,
                                          __nv_bfloat16* __restrict__ dlogits) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  for (int s = blockIdx.x * wpb + warp; s < S; s += gridDim.x * wpb) {
    float w = lane < K ? weights[(size_t)s * K + lane] : 0.f;
    float dw = lane < K ? dweights[(size_t)s * K + lane] : 0.f;
    float dot = w * dw;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    __nv_bfloat16* row = dlogits + (size_t)s * E;
    for (int e = lane; e < E; e += 32) row[e] = __float2bfloat16(0.f);
    __syncwarp();
    if (lane < K) row[topk[(size_t)s * K + lane]] = __float2bfloat16(w * (dw - dot));
  }
}

// ---- SwiGLU backward ----------------------------------------------------------------------------
// act = silu(g) * u * w  =>  dg = dact * u * w * silu'(g), du = dact * silu(g) * w,
//                            dw = sum_h dact * silu(g) * u
// One warp a row, whose lanes take its 16-byte vectors in turn, SB_DEPTH at once.  Bound by HBM (five bf16 tensors) and,
// next to it, by issue.  A block a row left 160 of 256 threads idle at H' = 768 and met at two barriers a row: 36900
// rows x 512 89 -> 46 us, x 2048 142 -> 134, 20000 x 1024 62 -> 48 (with the clearing of the sums in front, which the
// kernel now does itself for the rows behind the last).  More vectors at once cost the registers of other warps (four:
// 185 us for x 2048).  Few rows leave warps idle instead, and a warp's steps over a wide row are a chain of loads: up
// to SB_WIDE rows a vector a block takes each (512 rows x 2048 15.4 -> 9.2 us, 2500 20.8 -> 18.8; 512 x 768 10.9 -> 8.2;
// 4000 x 2048, above the line, 23.6 either way).  A row's sum has the same order either way: eight partial sums, of
// the vectors with the same v / 32 % 8, each over the lanes first.
constexpr int SB_WARPS = 8, SB_DEPTH = 2, SB_WIDE = 12;

struct SwigluRow {
  const uint4 *d, *g, *u;
  uint4 *dg, *du;
  float w;
  __device__ __forceinline__ SwigluRow(const __nv_bfloat16* dact, const __nv_bfloat16* gate, const __nv_bfloat16* up,
                                       __nv_bfloat16* dgate, __nv_bfloat16* dup, const float* row_scale, int r, int Hp)
      : d((const uint4*)(dact + (size_t)r * Hp)), g((const uint4*)(gate + (size_t)r * Hp)), u((const uint4*)(up + (size_t)r * Hp)),
        dg((uint4*)(dgate + (size_t)r * Hp)), du((uint4*)(dup + (size_t)r * Hp)), w(row_scale ? row_scale[r] : 1.f) {}
  // gradients of vector v; its terms of the row's sum are added to acc
  __device__ __forceinline__ void vec(int v, const uint4& d4, const uint4& g4, const uint4& u4, float& acc) const {
    uint4 rg, ru;
    const __nv_bfloat162* d2 = reinterpret_cast<const __nv_bfloat162*>(&d4);
    const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&g4);
    const __nv_bfloat162* u2 = reinterpret_cast<const __nv_bfloat162*>(&u4);
    __nv_bfloat162* og2 = reinterpret_cast<__nv_bfloat162*>(&rg);
    __nv_bfloat162* ou2 = reinterpret_cast<__nv_bfloat162*>(&ru);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 x = __bfloat1622float2(d2[e]), y = __bfloat1622float2(g2[e]), z = __bfloat1622float2(u2[e]);
      float s0 = 1.f / (1.f + __expf(-y.x)), s1 = 1.f / (1.f + __expf(-y.y));
      float sg0 = y.x * s0, sg1 = y.y * s1;
      acc += x.x * sg0 * z.x + x.y * sg1 * z.y;
      float dg0 = x.x * z.x * w * (s0 * (1.f + y.x * (1.f - s0)));
      float dg1 = x.y * z.y * w * (s1 * (1.f + y.y * (1.f - s1)));
      og2[e] = __floats2bfloat162_rn(dg0, dg1);
      ou2[e] = __floats2bfloat162_rn(x.x * sg0 * w, x.y * sg1 * w);
    }
    dg[v] = rg;
    du[v] = ru;
  }
};
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__global__ void __launch_bounds__(SB_WARPS * 32, 4)
ep_swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dact, const __nv_bfloat16* __restrict__ gate,
                     const __nv_bfloat16* __restrict__ up, const float* __restrict__ row_scale,
                     const int32_t* __restrict__ rows_ptr, int max_rows, int Hp,
                     __nv_bfloat16* __restrict__ dgate, __nv_bfloat16* __restrict__ dup,
                     float* __restrict__ dscale) {
  __shared__ float red[SB_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows = rows_ptr ? min(*rows_ptr, max_rows) : max_rows;
  const int nvec = Hp / 8;
  if (rows <= SB_WIDE * nvec) {
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
      const SwigluRow row(dact, gate, up, dgate, dup, row_scale, r, Hp);
      float part = 0.f;
      for (int v = threadIdx.x; v < nvec; v += SB_WARPS * 32) row.vec(v, row.d[v], row.g[v], row.u[v], part);
      if (dscale) {
        part = warp_sum(part);
        if (lane == 0) red[warp] = part;
        __syncthreads();
        if (threadIdx.x == 0)
          dscale[r] = ((red[0] + red[4]) + (red[2] + red[6])) + ((red[1] + red[5]) + (red[3] + red[7]));
        __syncthreads();
      }
    }
  } else {
    for (int r = blockIdx.x * SB_WARPS + warp; r < rows; r += gridDim.x * SB_WARPS) {
      const SwigluRow row(dact, gate, up, dgate, dup, row_scale, r, Hp);
      float part[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) part[i] = 0.f;
      for (int v0 = 0; v0 < nvec; v0 += 8 * 32) {
#pragma unroll
        for (int h = 0; h < 8; h += SB_DEPTH) {
          if (v0 + h * 32 >= nvec) break;
          uint4 d4[SB_DEPTH], g4[SB_DEPTH], u4[SB_DEPTH];
#pragma unroll
          for (int i = 0; i < SB_DEPTH; ++i) {
            const int v = v0 + (h + i) * 32 + lane;
            if (v < nvec) { d4[i] = row.d[v]; g4[i] = row.g[v]; u4[i] = row.u[v]; }
          }
#pragma unroll
          for (int i = 0; i < SB_DEPTH; ++i) {
            const int v = v0 + (h + i) * 32 + lane;
            if (v < nvec) row.vec(v, d4[i], g4[i], u4[i], part[h + i]);
          }
        }
      }
      if (dscale) {
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i] = warp_sum(part[i]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < o; ++i) part[i] += part[i + o];
        if (lane == 0) dscale[r] = part[0];
      }
    }
  }
  // rows that hold nothing
  if (dscale)
    for (int r = max(rows, 0) + blockIdx.x * SB_WARPS * 32 + threadIdx.x; r < max_rows; r += gridDim.x * SB_WARPS * 32) dscale[r] = 0.f;
}

// ---- cross-entropy over bf16 logits ---------------------------------------------------------------
// Forward: one block a row, one pass: every thread keeps a running maximum and the sum of exp(x - max)
// (fp32; rescaled when the maximum grows), the block combines them into the row's log-sum-exp.
// Backward: one pass, d logits = (exp(x - lse) - [x is the target]) * g / rows, rounded to bf16 once.
// The logits are read once each way and nothing of their size is written but the gradient; as
// cross_entropy(logits.float()) the same took an fp32 copy, two more fp32 tensors of their size and a
// copy back.  Bound by HBM: 4096 x 32000 logits are 262 MB, 40 us forward (read) and 80 us backward (read, and as
// much gradient written) at the copy rate.
constexpr int CE_THREADS = 512;

__device__ __forceinline__ void ce_add(float& m, float& s, float x) {
  // (m = -inf: s is 0 and exp(-inf) is 0; x - x is 0, or NaN for an infinite logit, as its loss is)
  if (x > m) { s = s * expf(m - x) + (1.f + (x - x)); m = x; }
  else if (!(x == -INFINITY && m == -INFINITY)) s += expf(x - m);
}

template <bool VEC>
__global__ void __launch_bounds__(CE_THREADS)
ep_ce_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, long long ignore,
                 int V, float* __restrict__ lse, float* __restrict__ loss) {
  __shared__ float sm[CE_THREADS / 32], ss[CE_THREADS / 32];
  const long long r = blockIdx.x;
  const __nv_bfloat16* row = logits + r * V;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float m = -INFINITY, s = 0.f;
  if constexpr (VEC) {
    const uint4* row4 = reinterpret_cast<const uint4*>(row);
    for (int v = threadIdx.x; v < V / 8; v += CE_THREADS) {
      const uint4 q = row4[v];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
      float x[8], top = -INFINITY;
#pragma unroll
      for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); x[2 * i] = f.x; x[2 * i + 1] = f.y; }
#pragma unroll
      for (int i = 0; i < 8; ++i) top = fmaxf(top, x[i]);
      if (top > m) { s *= expf(m - top); m = top; }
      if (m != -INFINITY) {
#pragma unroll
        for (int i = 0; i < 8; ++i) s += expf(x[i] - m);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) if (x[i] != x[i]) s = x[i];      // a NaN among nothing but -inf
      }
    }
  } else {
    for (int i = threadIdx.x; i < V; i += CE_THREADS) ce_add(m, s, __bfloat162float(row[i]));
  }
  auto join = [](float& m1, float& s1, float m2, float s2) {
    const float top = fmaxf(m1, m2);
    s1 = (s1 != 0.f ? s1 * (m1 == top ? 1.f : expf(m1 - top)) : 0.f) + (s2 != 0.f ? s2 * (m2 == top ? 1.f : expf(m2 - top)) : 0.f);
    m1 = top;
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) join(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  if (lane == 0) { sm[warp] = m; ss[warp] = s; }
  __syncthreads();
  if (warp == 0) {
    m = lane < CE_THREADS / 32 ? sm[lane] : -INFINITY;
    s = lane < CE_THREADS / 32 ? ss[lane] : 0.f;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) join(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
    if (lane == 0) {
      const float l = m + logf(s);
      const long long t = targets[r];
      lse[r] = l;
      // (a target that is no class: ep_ce_mean_kernel reports it)
      loss[r] = t == ignore ? 0.f : (t >= 0 && t < V ? l - __bfloat162float(row[t]) : NAN);
    }
  }
}

// out[0] = mean loss of the rows that count, out[1] = their number; summed in a fixed order.  A target that is
// no class makes both NaN, so that every gradient is too, and the first such row is recorded in `status`.
__global__ void __launch_bounds__(1024) ep_ce_mean_kernel(const float* __restrict__ loss, const long long* __restrict__ targets,
                                                         long long ignore, int S, int V, float* __restrict__ out,
                                                         int32_t* __restrict__ status) {
  __shared__ double sl[32];
  __shared__ int sn[32], sb[32];
  double l = 0.0;
  int n = 0, bad = S;
  for (int r = threadIdx.x; r < S; r += 1024) {
    const long long t = targets[r];
    l += loss[r];
    n += t != ignore;
    if (t != ignore && (t < 0 || t >= V)) bad = min(bad, r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
    bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, o));
  }
  if ((threadIdx.x & 31) == 0) { sl[threadIdx.x >> 5] = l; sn[threadIdx.x >> 5] = n; sb[threadIdx.x >> 5] = bad; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 32; ++i) { l += sl[i]; n += sn[i]; bad = min(bad, sb[i]); }
    out[0] = (float)(l / n);             // (no row counts: 0 / 0, NaN)
    out[1] = bad < S ? NAN : (float)n;
    if (bad < S && atomicCAS(status, 0, (int)ST_BAD_INDEX) == 0) {
      status[1] = KID_CROSS_ENTROPY;
      status[4] = bad;
      status[5] = (int)targets[bad];
      status[6] = V;
    }
  }
}

template <bool VEC>
__global__ void __launch_bounds__(CE_THREADS)
ep_ce_bwd_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, long long ignore,
                 int V, const float* __restrict__ lse, const float* __restrict__ mean_n, const float* __restrict__ g,
                 __nv_bfloat16* __restrict__ grad) {
  const long long r = blockIdx.x;
  const __nv_bfloat16* row = logits + r * V;
  __nv_bfloat16* out = grad + r * V;
  const long long t = targets[r];
  const bool counts = t != ignore;
  const float l = lse[r], scale = counts ? g[0] / mean_n[1] : 0.f;
  auto d = [&](float x, int i) { return counts ? (expf(x - l) - (i == t ? 1.f : 0.f)) * scale : 0.f; };
  if constexpr (VEC) {
    for (int v = threadIdx.x; v < V / 8; v += CE_THREADS) {
      uint4 q = reinterpret_cast<const uint4*>(row)[v];
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        h[i] = __floats2bfloat162_rn(d(f.x, 8 * v + 2 * i), d(f.y, 8 * v + 2 * i + 1));
      }
      reinterpret_cast<uint4*>(out)[v] = q;
    }
  } else {
    for (int i = threadIdx.x; i < V; i += CE_THREADS) out[i] = __float2bfloat16(d(__bfloat162float(row[i]), i));
  }
}

// ---- SGD: w(bf16) -= lr * g(fp32) ----------------------------------------------------------------
// Bound by HBM: 8 bytes a weight, 6.8 TB/s.  A layer's tensors are one launch, whose threads stride on from one tensor
// into the next: a launch each left the device idle three times between them (a whole step of 32 experts, 1024 x 512: 564 -> 538 us).
constexpr int SGD_TENSORS = 8;
struct SgdTensors {
  __nv_bfloat16* w[SGD_TENSORS];
  const float* g[SGD_TENSORS];
  long long n[SGD_TENSORS];
  int count;
};

__device__ __forceinline__ void sgd_vec(__nv_bfloat16* w, const float* g, long long v, float nlr) {
  uint4 w4 = reinterpret_cast<uint4*>(w)[v];
  float4 g0 = reinterpret_cast<const float4*>(g)[2 * v], g1 = reinterpret_cast<const float4*>(g)[2 * v + 1];
  __nv_bfloat162* w2 = reinterpret_cast<__nv_bfloat162*>(&w4);
  const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 x = __bfloat1622float2(w2[i]);
    w2[i] = __floats2bfloat162_rn(__fmaf_rn(nlr, gg[2 * i], x.x), __fmaf_rn(nlr, gg[2 * i + 1], x.y));
  }
  reinterpret_cast<uint4*>(w)[v] = w4;
}

__global__ void __launch_bounds__(256) ep_sgd_kernel(const __grid_constant__ SgdTensors t, float lr) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const float nlr = -lr;
  long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = 0; i < t.count; ++i) {
    __nv_bfloat16* w = t.w[i];
    const float* __restrict__ g = t.g[i];
    const long long n = t.n[i], nvec = n / 8;
    for (; v < nvec; v += stride) sgd_vec(w, g, v, nlr);
    v -= nvec;
    if (blockIdx.x == 0 && threadIdx.x == 0)
      for (long long e = nvec * 8; e < n; ++e) w[e] = __float2bfloat16(__fmaf_rn(nlr, g[e], __bfloat162float(w[e])));
  }
}

// blockIdx.y is the expert; experts with a zero flag were updated elsewhere
__global__ void __launch_bounds__(256)
ep_sgd_masked_kernel(__nv_bfloat16* w, const float* __restrict__ g, float lr, const int32_t* __restrict__ only,
                     long long vec_per_expert) {
  if (only[blockIdx.y] == 0) return;
  const long long stride = (long long)gridDim.x * blockDim.x, v1 = (long long)(blockIdx.y + 1) * vec_per_expert;
  for (long long v = (long long)blockIdx.y * vec_per_expert + (long long)blockIdx.x * blockDim.x + threadIdx.x; v < v1; v += stride)
    sgd_vec(w, g, v, -lr);
}

}  // namespace mep

using namespace mep;

extern "C" {

int mep_router_topk(const float* logits, const float* bias, int S, int E, int K, int32_t* topk,
                    float* weights, int32_t* tpe, cudaStream_t stream) {
  if (K > 32 || K < 1 || E < K) return fail(-1, "router: need 1 <= K <= min(32, E)");
  // as many warps a block as its keys leave room for (up to 256 experts they are in registers)
  int warps = ROUTER_WARPS;
  if (E > 32 * ROUTER_VPL) {
    const int room = (int)(200 * 1024 / (sizeof(uint32_t) * (size_t)E)) - 1;
    if (room < 1) return fail(-2, "router: E=%d too large", E);
    if (room < warps) warps = room;
  }
  int blocks = (S + warps - 1) / warps;
  const int most = 148 * (E <= 32 * ROUTER_VPL ? 2 : (E <= 1536 ? 4 : (E <= 2816 ? 2 : 1)));
  if (blocks > most) blocks = most;
  MEP_CUDA_OK(cudaMemsetAsync(tpe, 0, sizeof(int32_t) * E, stream));
  if (E <= 32 * ROUTER_VPL) {
    ep_router_topk_kernel<true><<<blocks, ROUTER_WARPS * 32, E * sizeof(uint32_t), stream>>>(logits, bias, S, E, K, topk, weights, tpe);
  } else {
    const size_t smem = (size_t)(warps + 1) * E * sizeof(uint32_t);
    static std::atomic<unsigned long long> raised{0};
    MEP_CUDA_OK(raise_smem_limit((const void*)ep_router_topk_kernel<false>, raised));
    ep_router_topk_kernel<false><<<blocks, warps * 32, smem, stream>>>(logits, bias, S, E, K, topk, weights, tpe);
  }
  MEP_CUDA_OK(cudaGetLastError());
  return 0;
}

int mep_router_topk_bwd(const float* weights, const float* dweights, const int32_t* topk, int S, int E,
                        int K, void* dlogits, cudaStream_t stream) {
  int blocks = (S + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  ep_router_topk_bwd_kernel<<<blocks, 256, 0, stream>>>(weights, dweights, topk, S, E, K,
                                                       (__nv_bfloat16*)dlogits);
  MEP_CUDA_OK(cudaGetLastError());
  return 0;
}

int mep_swiglu_bwd(const void* dact, const void* gate, const void* up, const float* row_scale,
                   const int32_t* rows_ptr, int max_rows, int Hp, void* dgate, void* dup,
                   float* dscale, cudaStream_t stream) {
  if (Hp % 8 != 0) return fail(-1, "swiglu_bwd: H'=%d must be a multiple of 8", Hp);
  // as many blocks as either way of taking rows can use
  const int wide = max_rows < SB_WIDE * (Hp / 8) ? max_rows : SB_WIDE * (Hp / 8);
  int blocks = (max_rows + SB_WARPS - 1) / SB_WARPS;
  if (blocks < wide) blocks = wide;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) return 0;
  ep_swiglu_bwd_kernel<<<blocks, SB_WARPS * 32, 0, stream>>>(
      (const __nv_bfloat16*)dact, (const __nv_bfloat16*)gate, (const __nv_bfloat16*)up, row_scale,
      rows_ptr, max_rows, Hp, (__nv_bfloat16*)dgate, (__nv_bfloat16*)dup, dscale);
  MEP_CUDA_OK(cudaGetLastError());
  return 0;
}

// logits [S][V] bf16, targets [S] int64; lse, loss [S] and mean_n [2] (mean, rows that count) fp32; status
// int32 [8], where a target that is neither `ignore` nor a class is recorded.
int mep_ce_fwd(const void* logits, const long long* targets, long long ignore, int S, int V, float* lse, float* loss,
               float* mean_n, int32_t* status, cudaStream_t stream) {
  if (V < 1 || S < 0) return fail(-1, "cross entropy: %d x %d logits", S, V);
  const __nv_bfloat16* x = (const __nv_bfloat16*)logits;
  if (S > 0) {
    if (V % 8 == 0 && (uintptr_t)logits % 16 == 0)
      ep_ce_fwd_kernel<true><<<S, CE_THREADS, 0, stream>>>(x, targets, ignore, V, lse, loss);
    else
      ep_ce_fwd_kernel<false><<<S, CE_THREADS, 0, stream>>>(x, targets, ignore, V, lse, loss);
  }
  ep_ce_mean_kernel<<<1, 1024, 0, stream>>>(loss, targets, ignore, S, V, mean_n, status);
  MEP_CUDA_OK(cudaGetLastError());
  return 0;
}

// grad [S][V] bf16 of g[0] * mean loss
int mep_ce_bwd(const void* logits, const long long* targets, long long ignore, int S, int V, const float* lse,
               const float* mean_n, const float* g, void* grad, cudaStream_t stream) {
  if (V < 1 || S < 0) return fail(-1, "cross entropy: %d x %d logits", S, V);
  if (S == 0) return 0;
  const __nv_bfloat16* x = (const __nv_bfloat16*)logits;
  __nv_bfloat16* out = (__nv_bfloat16*)grad;
  if (V % 8 == 0 && (((uintptr_t)logits | (uintptr_t)grad) % 16) == 0)
    ep_ce_bwd_kernel<true><<<S, CE_THREADS, 0, stream>>>(x, targets, ignore, V, lse, mean_n, g, out);
  else
    ep_ce_bwd_kernel<false><<<S, CE_THREADS, 0, stream>>>(x, targets, ignore, V, lse, mean_n, g, out);
  MEP_CUDA_OK(cudaGetLastError());
  return 0;
}

// Tensors i < count: w[i] bf16 [n[i]] -= lr * g[i] fp32 [n[i]].
int mep_sgd_update(void* const* w, const void* const* g, const long long* n, int count, float lr, cudaStream_t stream) {
  if (count < 1 || count > SGD_TENSORS) return fail(-2, "sgd: 1..%d tensors in a launch", SGD_TENSORS);
  SgdTensors t;
  long long nvec = 0;
  for (int i = 0; i < count; ++i) {
    if (((uintptr_t)w[i] | (uintptr_t)g[i]) % 16 != 0) return fail(-1, "sgd: tensors must be 16-byte aligned");
    t.w[i] = (__nv_bfloat16*)w[i]; t.g[i] = (const float*)g[i]; t.n[i] = n[i];
    nvec += n[i] / 8;
  }
  t.count = count;
  long long blocks = (nvec + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) blocks = 1;
  ep_sgd_kernel<<<(int)blocks, 256, 0, stream>>>(t, lr);
  MEP_CUDA_OK(cudaGetLastError());
  return 0;
}

// Same update, restricted to the experts whose flag is non-zero: w and g are [experts][elems].
int mep_sgd_update_masked(void* w, const float* g, long long experts, long long elems, const int32_t* only,
                          float lr, cudaStream_t stream) {
  if (((uintptr_t)w | (uintptr_t)g) % 16 != 0 || elems % 8 != 0)
    return fail(-1, "sgd: tensors must be 16-byte aligned and elems a multiple of 8");
  if (experts < 1 || experts > 65535) return fail(-2, "sgd: 1..65535 experts");
  long long nvec = elems / 8;
  long long blocks = (nvec + 255) / 256;
  if (blocks > 148 * 4) blocks = 148 * 4;
  if (blocks < 1) blocks = 1;
  ep_sgd_masked_kernel<<<dim3((unsigned)blocks, (unsigned)experts), 256, 0, stream>>>((__nv_bfloat16*)w, g, lr, only, nvec);
  MEP_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // extern "C"
