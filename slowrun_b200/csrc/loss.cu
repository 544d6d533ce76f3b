// Soft-capped cross-entropy over bf16 logits, forward and backward in one kernel: one CTA per token row,
// pass 1 = online max/sum of z = cap*tanh(x/cap), pass 2 (row is L2 resident) writes
// dlogits = scale * (S_w * softmax(z) - sum_k w_k onehot(y_k)) * (1 - tanh^2) in place as bf16.
// Supports the shifted-target multi-token loss of the tiny track (weights w_k for targets at flattened
// index row+k, tiny/cuda_kernels.py:226-240) and ignore_index = -1. The reference computes the limited-track
// loss with fp32 logits through Inductor (train.py:559-564) and the tiny one with its NVRTC kernel.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace {

constexpr int kThreads = 256;
constexpr int kMaxPredict = 4;

struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

// z = cap * tanh(x / cap) with the hardware tanh (one special-function op; its 2^-11 relative error is an eighth of
// the bf16 quantisation of the logits themselves). The kernel is bound by the special-function pipe, so the softcap
// costs one op instead of the two of an exp + reciprocal formulation.
__device__ __forceinline__ float softcap(float x, float cap, float inv_cap, float& t) {
  if (cap <= 0.f) {
    t = 0.f;
    return x;
  }
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x * inv_cap));
  return cap * t;
}

__global__ void __launch_bounds__(kThreads)
softcap_ce_kernel(__nv_bfloat16* __restrict__ logits, const long* __restrict__ targets, float* __restrict__ loss,
                  const float* __restrict__ weights, int n_predict, const float* __restrict__ scale_ptr, long M,
                  int Vpad, int V, long ld, float cap, int write_grad) {
  __shared__ float red_m[kThreads / 32], red_s[kThreads / 32];
  __shared__ float sh_lse;
  const long row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const float inv_cap = cap > 0.f ? 1.f / cap : 0.f;

  long tgt[kMaxPredict];
  float w[kMaxPredict];
  float sw = 0.f;
  for (int k = 0; k < kMaxPredict; ++k) {
    tgt[k] = -1;
    w[k] = 0.f;
    if (k < n_predict && row + k < M) {
      const long y = targets[row + k];
      const float wk = weights ? weights[k] : 1.f;
      if (y >= 0 && y < V && wk != 0.f) {
        tgt[k] = y;
        w[k] = wk;
        sw += wk;
      }
    }
  }
  if (sw == 0.f && n_predict == 1) {
    // ignored row: zero loss, zero gradient
    if (threadIdx.x == 0) loss[row] = 0.f;
    if (write_grad) {
      bf16x8 z;
      for (int i = 0; i < 4; ++i) z.v[i] = __floats2bfloat162_rn(0.f, 0.f);
      for (int c = threadIdx.x * 8; c < Vpad; c += kThreads * 8) *reinterpret_cast<bf16x8*>(lr + c) = z;
    }
    return;
  }

  // pass 1: online max / sum over the valid vocabulary
  float m = cap > 0.f ? cap : -INFINITY, s = 0.f;
  for (int c = threadIdx.x * 8; c < Vpad; c += kThreads * 8) {
    const bf16x8 v = *reinterpret_cast<const bf16x8*>(lr + c);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(v.v[i]);
      float t;
      if (c + 2 * i < V) {
        const float z = softcap(f.x, cap, inv_cap, t);
        if (cap > 0.f) {          // |z| <= cap: the bound serves as the maximum, exp(z - cap) >= exp(-2 cap)
          s += __expf(z - cap);
        } else if (z > m) {
          s = s * __expf(m - z) + 1.f;
          m = z;
        } else {
          s += __expf(z - m);
        }
      }
      if (c + 2 * i + 1 < V) {
        const float z = softcap(f.y, cap, inv_cap, t);
        if (cap > 0.f) {
          s += __expf(z - cap);
        } else if (z > m) {
          s = s * __expf(m - z) + 1.f;
          m = z;
        } else {
          s += __expf(z - m);
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
    const float mm = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * __expf(m - mm)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mm));
    m = mm;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    red_m[warp] = m;
    red_s[warp] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mm = red_m[0], ss = red_s[0];
    for (int i = 1; i < kThreads / 32; ++i) {
      const float m2 = red_m[i], s2 = red_s[i];
      const float mx = fmaxf(mm, m2);
      ss = (mm == -INFINITY ? 0.f : ss * __expf(mm - mx)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mx));
      mm = mx;
    }
    const float lse = mm + logf(ss);
    sh_lse = lse;
    float l = 0.f;
    for (int k = 0; k < kMaxPredict; ++k) {
      if (tgt[k] >= 0) {
        float t;
        const float z = softcap(__bfloat162float(lr[tgt[k]]), cap, inv_cap, t);
        l += w[k] * (lse - z);
      }
    }
    loss[row] = l;
  }
  if (!write_grad) return;
  __syncthreads();
  const float lse = sh_lse;
  const float scale = scale_ptr ? *scale_ptr : 1.f;

  // pass 2: gradient in place
  for (int c = threadIdx.x * 8; c < Vpad; c += kThreads * 8) {
    bf16x8 v = *reinterpret_cast<const bf16x8*>(lr + c);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(v.v[i]);
      float g[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = c + 2 * i + e;
        float t;
        const float z = softcap(e ? f.y : f.x, cap, inv_cap, t);
        float gv = 0.f;
        if (col < V) {
          gv = sw * __expf(z - lse);
#pragma unroll
          for (int k = 0; k < kMaxPredict; ++k)
            if (tgt[k] == col) gv -= w[k];
          gv *= scale * (1.f - t * t);
        }
        g[e] = gv;
      }
      v.v[i] = __floats2bfloat162_rn(g[0], g[1]);
    }
    *reinterpret_cast<bf16x8*>(lr + c) = v;
  }
}

// ---------------------------------------------------------------------------------------------- logits as an output
// z = cap * tanh(x / cap) of the first V columns, fp32, and its backward. Bound by memory: one pass instead of the copy,
// division, tanh and product of the op-by-op form (4 reads and 4 writes of the fp32 logits).
// [4096, 50257]: 345 us forward and 335 us backward against about 2900 us and 2000 us op by op.
// tanh(u) = e / (e + 2) with e = expm1(2u): full fp32 precision also near 0, unlike the hardware tanh used above. Both
// quotients are an approximate one plus a correction by its residual, a fraction of the instructions of an IEEE division.
__device__ __forceinline__ float quotient(float x, float d, float r) {   // x / d, r = 1 / d to a few units in the last place
  const float q = x * r;
  return fmaf(fmaf(-q, d, x), r, q);
}
__device__ __forceinline__ float softcap_exact(float x, float cap, float inv_cap) {
  const float u = quotient(x, cap, inv_cap);
  const float e = expm1f(2.f * fminf(fabsf(u), 20.f));    // tanh(20) rounds to 1
  const float t = quotient(e, e + 2.f, __fdividef(1.f, e + 2.f));
  return cap * copysignf(u != u ? u : t, u);
}

__global__ void __launch_bounds__(kThreads)
softcap_logits_fwd_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ z, int V, long ld, float cap) {
  const long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * ld;
  float* zr = z + row * V;
  const float inv_cap = cap > 0.f ? 1.f / cap : 0.f;
#pragma unroll 4
  for (int c = threadIdx.x; c < V; c += kThreads) {
    const float v = __bfloat162float(xr[c]);
    zr[c] = cap > 0.f ? softcap_exact(v, cap, inv_cap) : v;
  }
}

// dx = g * (1 - (z / cap)^2), zero in the padding columns
__global__ void __launch_bounds__(kThreads)
softcap_logits_bwd_kernel(const float* __restrict__ g, const float* __restrict__ z, __nv_bfloat16* __restrict__ dx, int V, int Vpad,
                          long ld, float cap) {
  const long row = blockIdx.x;
  const float *gr = g + row * V, *zr = z + row * V;
  __nv_bfloat16* dr = dx + row * ld;
  const float inv_cap = cap > 0.f ? 1.f / cap : 0.f;
#pragma unroll 4
  for (int c = threadIdx.x; c < Vpad; c += kThreads) {
    float d = 0.f;
    if (c < V) {
      const float t = zr[c] * inv_cap;
      d = gr[c] * (1.f - t * t);
    }
    dr[c] = __float2bfloat16(d);
  }
}

// ---------------------------------------------------------------------------------------------- distillation
// Cross-entropy (label smoothing `ls`) and KL(teacher / T || student / T) of fp32 logits, one CTA per row, and their
// gradient. The rows are read twice in the forward (the second time from L2) and once in the backward; nothing of the size
// of the logits is written but the gradient. [4096, 50257]: 560 us forward and 395 us backward against about 10 ms op by op.
constexpr int kDistThreads = 512;

struct MaxSum {   // sum of exp(v - m) over what has been seen; m = maximum
  float m, s;
};
__device__ __forceinline__ float exp_nat(float x) { return exp2f(x * 1.4426950408889634f); }
__device__ __forceinline__ void add_value(MaxSum& a, float v) {
  if (v > a.m) {
    a.s = a.s * exp_nat(a.m - v) + 1.f;
    a.m = v;
  } else {
    a.s += exp_nat(v - a.m);
  }
}
__device__ __forceinline__ MaxSum merge(MaxSum a, MaxSum b) {
  const float m = fmaxf(a.m, b.m);
  return MaxSum{m, (a.m == -INFINITY ? 0.f : a.s * exp_nat(a.m - m)) + (b.m == -INFINITY ? 0.f : b.s * exp_nat(b.m - m))};
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  __syncthreads();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < kDistThreads / 32; ++i) t += red[i];
  return t;
}
__device__ __forceinline__ float block_lse(MaxSum v, MaxSum* red) {
  __syncthreads();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = merge(v, MaxSum{__shfl_xor_sync(0xffffffffu, v.m, o), __shfl_xor_sync(0xffffffffu, v.s, o)});
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  MaxSum t = red[0];
  for (int i = 1; i < kDistThreads / 32; ++i) t = merge(t, red[i]);
  return t.m + static_cast<float>(log(static_cast<double>(t.s)));   // once per row; the fast single-precision log is off by 2^-21
}

// stats: [3, M] log-sum-exp of s, s / T and t / T; ce, kl: [M] (0 for ignored rows)
__global__ void __launch_bounds__(kDistThreads)
distill_fwd_kernel(const float* __restrict__ s, const float* __restrict__ t, const long* __restrict__ y, float* __restrict__ ce,
                   float* __restrict__ kl, float* __restrict__ stats, long M, int V, float inv_T, float ls) {
  __shared__ MaxSum red[kDistThreads / 32];
  __shared__ float red1[kDistThreads / 32];
  const long row = blockIdx.x;
  const long target = y[row];
  if (target == -1) {
    if (threadIdx.x == 0) ce[row] = kl[row] = stats[row] = stats[M + row] = stats[2 * M + row] = 0.f;
    return;
  }
  const float *sr = s + row * V, *tr = t + row * V;
  const bool same = inv_T == 1.f;
  MaxSum a{-INFINITY, 0.f}, b{-INFINITY, 0.f}, c{-INFINITY, 0.f};
  float sum = 0.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < V; i += kDistThreads) {
    const float x = sr[i], u = tr[i];
    add_value(a, x);
    if (!same) add_value(b, x * inv_T);
    add_value(c, u * inv_T);
    sum += x;
  }
  const float l1 = block_lse(a, red), lt = block_lse(c, red), lT = same ? l1 : block_lse(b, red);
  float k = 0.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < V; i += kDistThreads) {
    const float lp = tr[i] * inv_T - lt;
    k += exp_nat(lp) * (lp - (sr[i] * inv_T - lT));
  }
  k = block_sum(k, red1);
  sum = ls > 0.f ? block_sum(sum, red1) : 0.f;
  if (threadIdx.x == 0) {
    const bool ok = target >= 0 && target < V;
    const float nll = ok ? l1 - sr[target] : __int_as_float(0x7fc00000);     // a target outside the vocabulary: NaN
    ce[row] = (1.f - ls) * nll + (ls > 0.f ? ls * (l1 - sum / (float)V) : 0.f);
    kl[row] = k;
    stats[row] = l1;
    stats[M + row] = lT;
    stats[2 * M + row] = lt;
  }
}

// ds = g_ce / N * (softmax(s) - target distribution) + g_kl / (N T) * (softmax(s / T) - softmax(t / T))
__global__ void __launch_bounds__(kDistThreads)
distill_bwd_kernel(const float* __restrict__ s, const float* __restrict__ t, const long* __restrict__ y, const float* __restrict__ stats,
                   const float* __restrict__ n_valid, const float* __restrict__ g_ce, const float* __restrict__ g_kl,
                   float* __restrict__ ds, long M, int V, float inv_T, float ls) {
  const long row = blockIdx.x;
  const long target = y[row];
  const float *sr = s + row * V, *tr = t + row * V;
  float* dr = ds + row * V;
  if (target == -1) {
    for (int i = threadIdx.x; i < V; i += kDistThreads) dr[i] = 0.f;
    return;
  }
  const float l1 = stats[row], lT = stats[M + row], lt = stats[2 * M + row];
  const float wc = *g_ce / *n_valid, wk = *g_kl / *n_valid * inv_T, base = ls / (float)V;
  const bool same = inv_T == 1.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < V; i += kDistThreads) {
    const float x = sr[i];
    const float p1 = exp_nat(x - l1), pT = same ? p1 : exp_nat(x * inv_T - lT), pt = exp_nat(tr[i] * inv_T - lt);
    const float q = base + (i == target ? 1.f - ls : 0.f);
    dr[i] = wc * (p1 - q) + wk * (pT - pt);
  }
}

}  // namespace

// logits: [M, ld] bf16 (ld >= Vpad, Vpad % 8 == 0), overwritten with the gradient when write_grad != 0.
// targets: int64 [M]; loss: fp32 [M]; weights: optional device fp32[n_predict]; scale_ptr: optional device scalar
// multiplied into the gradient (e.g. 1 / number of valid tokens).
extern "C" int sr_softcap_ce(void* logits, const long* targets, float* loss, const float* weights, int n_predict,
                             const float* scale_ptr, long M, int Vpad, int V, long ld, float cap, int write_grad,
                             cudaStream_t s) {
  if (M <= 0) return 0;
  if (Vpad % 8 || ld % 8 || n_predict < 1 || n_predict > kMaxPredict || V > Vpad) return -2;
  softcap_ce_kernel<<<(unsigned)M, kThreads, 0, s>>>(reinterpret_cast<__nv_bfloat16*>(logits), targets, loss, weights,
                                                     n_predict, scale_ptr, M, Vpad, V, ld, cap, write_grad);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// x: bf16 [M, ld]; z: fp32 [M, V] contiguous. cap <= 0: z = x.
extern "C" int sr_softcap_logits_fwd(const void* x, float* z, long M, int V, long ld, float cap, cudaStream_t s) {
  if (M <= 0 || V <= 0) return 0;
  if (ld < V || M > 0x7fffffffL) return -2;
  softcap_logits_fwd_kernel<<<(unsigned)M, kThreads, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), z, V, ld, cap);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
// g, z: fp32 [M, V] contiguous; dx: bf16 [M, ld], columns 0 .. Vpad - 1 written.
extern "C" int sr_softcap_logits_bwd(const float* g, const float* z, void* dx, long M, int V, int Vpad, long ld, float cap, cudaStream_t s) {
  if (M <= 0 || Vpad <= 0) return 0;
  if (ld < Vpad || V > Vpad || M > 0x7fffffffL) return -2;
  softcap_logits_bwd_kernel<<<(unsigned)M, kThreads, 0, s>>>(g, z, reinterpret_cast<__nv_bfloat16*>(dx), V, Vpad, ld, cap);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
// s, t: fp32 [M, V] contiguous; y: int64 [M], -1 = ignored; ce, kl: fp32 [M]; stats: fp32 [3, M].
extern "C" int sr_distill_fwd(const float* s, const float* t, const long* y, float* ce, float* kl, float* stats, long M, int V, float T,
                              float label_smoothing, cudaStream_t st) {
  if (M <= 0) return 0;
  if (V <= 0 || M > 0x7fffffffL) return -2;
  distill_fwd_kernel<<<(unsigned)M, kDistThreads, 0, st>>>(s, t, y, ce, kl, stats, M, V, 1.f / T, label_smoothing);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
// n_valid, g_ce, g_kl: device fp32 scalars (number of rows that count; gradients of the two means); ds: fp32 [M, V].
extern "C" int sr_distill_bwd(const float* s, const float* t, const long* y, const float* stats, const float* n_valid, const float* g_ce,
                              const float* g_kl, float* ds, long M, int V, float T, float label_smoothing, cudaStream_t st) {
  if (M <= 0) return 0;
  if (V <= 0 || M > 0x7fffffffL) return -2;
  distill_bwd_kernel<<<(unsigned)M, kDistThreads, 0, st>>>(s, t, y, stats, n_valid, g_ce, g_kl, ds, M, V, 1.f / T, label_smoothing);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
