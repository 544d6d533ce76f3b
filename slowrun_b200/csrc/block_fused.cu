// Kernels that exist only because the transformer block is executed as ONE autograd node with a hand-written
// backward (slowrun_b200/ops/block.py): every gradient buffer is written exactly once, so no slice/concat/zero-fill
// glue is left to the autograd engine.
//
//   qkv_prep fwd/bwd   split the fused [M, 3d] projection, add the gated value residual to v, apply RoPE and the
//                      per-head RMSNorm to q and k; backward writes one dense dqkv buffer (train.py:296-306).
//                      With `key_offset` the upper half of every key vector is the one computed for the previous token
//                      of the same sequence (token 0 keeps its own): the tiny track's partial key offset on
//                      long-window layers (tiny/train.py:447-449), done as a shifted store / shifted gradient load.
//   attn_post fwd/bwd  what follows the attention kernel per (token, head): exclusive self-attention
//                      y -= tanh(alpha_h) (y . v^) v^ with v^ the normalised value vector of the same token
//                      (tiny/train.py:451-458), then the per-head sigmoid gate (train.py:308-309). The backward also
//                      emits the attention backward's `delta` = rowsum(dO * O), the XSA contribution to dV and the
//                      gradient of alpha.
//   iha_mix fwd/bwd    Interleaved-head mixing of projection weights W'[h] = sum_m mix[h,m] W[m] on bf16 shadows and
//                      its gradients (dW += mix^T dW', dmix = dW' W^T). The reference leaves the [H, d*D] x [d*D, H]
//                      product to a library GEMM (train.py:277-280); with H <= 20 that is a long skinny reduction,
//                      done here as a streaming kernel plus a shared-memory tree.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <initializer_list>

namespace {

constexpr int kWarpsPerBlock = 8;
constexpr int kThreads = kWarpsPerBlock * 32;

inline int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

__device__ __forceinline__ float2 ld2(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}
__device__ __forceinline__ void st2(__nv_bfloat16* p, float a, float b) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}

// ---------------------------------------------------------------------------------------------- per-head vectors
// The kernels below work on (token, head) vectors of 128 elements. Eight lanes hold one: lane l has elements 8l .. 8l+7 and
// 64+8l .. 64+8l+7, i.e. both partners of its rotary pairs, in two 16-byte accesses per tensor. A warp then has four vectors
// in flight and a reduction is six or twelve shuffles for the four of them; with a warp per vector it was five shuffles each
// and 4-byte accesses, and the kernels were bound by instructions. us, warp per vector -> this, [8192, 20 heads]: qkv_prep fwd
// 76 -> 50, bwd 114 -> 88, attn_post bwd 57 -> 37; [65536, 8 heads]: 217 -> 158, 342 -> 293, 272 -> 187, attn_post fwd 101 -> 67.
constexpr int kVecPerBlock = kThreads / 8;

struct Vec {
  float lo[8], hi[8];
};
__device__ __forceinline__ void unpack8(const uint4& t, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&t);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = __bfloat1622float2(h[i]);
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}
__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float (&f)[8]) { unpack8(*reinterpret_cast<const uint4*>(p), f); }
__device__ __forceinline__ void st8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 t;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&t);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = t;
}
__device__ __forceinline__ void ldf8(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
  f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
// p: first element of the vector; l: lane within the eight
__device__ __forceinline__ Vec ldv(const __nv_bfloat16* p, int l) {
  Vec v;
  ld8(p + 8 * l, v.lo);
  ld8(p + 64 + 8 * l, v.hi);
  return v;
}
__device__ __forceinline__ void stv(__nv_bfloat16* p, int l, const Vec& v) {
  st8(p + 8 * l, v.lo);
  st8(p + 64 + 8 * l, v.hi);
}
// sum over the eight lanes of a vector
__device__ __forceinline__ float sum8(float v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The sums keep the order of a butterfly over 32 lanes, so that results do not depend on how many lanes share a vector: a
// change of rounding travels through every later layer and shows as 1 to 2 % in gradients that are sums with cancellation. Lane l stands for lanes 4l .. 4l+3 of a warp with elements {2L, 2L+1, 64+2L, 64+2L+1} each
// (dot_pairs) or for lanes 2l, 2l+1, 16+2l, 16+2l+1 with elements 4L .. 4L+3 (dot_quads).
__device__ __forceinline__ float dot_pairs(const Vec& a, const Vec& b) {
  float s[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    s[j] = a.lo[2 * j] * b.lo[2 * j] + a.lo[2 * j + 1] * b.lo[2 * j + 1] + a.hi[2 * j] * b.hi[2 * j] + a.hi[2 * j + 1] * b.hi[2 * j + 1];
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = sum8(s[j]);
  return (s[0] + s[2]) + (s[1] + s[3]);
}
__device__ __forceinline__ float dot_quads(const Vec& a, const Vec& b) {
  float s[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int i = 4 * j;
    const float lo = a.lo[i] * b.lo[i] + a.lo[i + 1] * b.lo[i + 1] + a.lo[i + 2] * b.lo[i + 2] + a.lo[i + 3] * b.lo[i + 3];
    const float hi = a.hi[i] * b.hi[i] + a.hi[i + 1] * b.hi[i + 1] + a.hi[i + 2] * b.hi[i + 2] + a.hi[i + 3] * b.hi[i + 3];
    s[j] = sum8(lo + hi);
  }
  return s[0] + s[1];
}

// ---------------------------------------------------------------------------------------------- qkv prep
__global__ void __launch_bounds__(kThreads)
qkv_prep_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ ve, const float* __restrict__ gate,
                    const __nv_bfloat16* __restrict__ cosb, const __nv_bfloat16* __restrict__ sinb, __nv_bfloat16* __restrict__ q_out,
                    __nv_bfloat16* __restrict__ k_out, __nv_bfloat16* __restrict__ v_out, unsigned n, unsigned H, unsigned T, float eps,
                    int key_offset) {
  const unsigned id = blockIdx.x * kVecPerBlock + (threadIdx.x >> 3);
  const bool valid = id < n;                      // the shuffles below want whole warps
  const unsigned vid = valid ? id : n - 1;
  const int l = threadIdx.x & 7;
  const unsigned tok = vid / H, h = vid - tok * H, t = tok % T;
  const long d = (long)H * 128;
  const __nv_bfloat16* in = qkv + (long)tok * 3 * d + h * 128;
  float c[8], s[8];
  ld8(cosb + (long)t * 64 + 8 * l, c);
  ld8(sinb + (long)t * 64 + 8 * l, s);
  const Vec x[2] = {ldv(in, l), ldv(in + d, l)};
  Vec v = ldv(in + 2 * d, l);
  if (ve != nullptr) {
    const float g = gate[vid];
    const Vec e = ldv(ve + (long)tok * d + h * 128, l);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v.lo[i] += g * e.lo[i];
      v.hi[i] += g * e.hi[i];
    }
  }
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    Vec o;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o.lo[i] = x[which].lo[i] * c[i] + x[which].hi[i] * s[i];
      o.hi[i] = -x[which].lo[i] * s[i] + x[which].hi[i] * c[i];
    }
    const float r = rsqrtf(dot_pairs(o, o) * (1.f / 128.f) + eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o.lo[i] *= r;
      o.hi[i] *= r;
    }
    if (valid) {
      __nv_bfloat16* p = (which == 0 ? q_out : k_out) + (long)vid * 128;
      st8(p + 8 * l, o.lo);
      if (which == 1 && key_offset) {
        // upper half goes to the next token of the sequence (same head: H vectors further); token 0 also keeps its own
        if (t + 1 < T) st8(p + d + 64 + 8 * l, o.hi);
        if (t == 0) st8(p + 64 + 8 * l, o.hi);
      } else {
        st8(p + 64 + 8 * l, o.hi);
      }
    }
  }
  if (valid) stv(v_out + (long)vid * 128, l, v);
}

__global__ void __launch_bounds__(kThreads)
qkv_prep_bwd_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ ve, const float* __restrict__ gate,
                    const __nv_bfloat16* __restrict__ cosb, const __nv_bfloat16* __restrict__ sinb, const __nv_bfloat16* __restrict__ dq,
                    const __nv_bfloat16* __restrict__ dk, const __nv_bfloat16* __restrict__ dv, __nv_bfloat16* __restrict__ dqkv,
                    __nv_bfloat16* __restrict__ dve, float* __restrict__ dgate, unsigned n, unsigned H, unsigned T, float eps,
                    const float* __restrict__ dq_f32, int key_offset, const __nv_bfloat16* __restrict__ dv_extra) {
  const unsigned id = blockIdx.x * kVecPerBlock + (threadIdx.x >> 3);
  const bool valid = id < n;
  const unsigned vid = valid ? id : n - 1;
  const int l = threadIdx.x & 7;
  const unsigned tok = vid / H, h = vid - tok * H, t = tok % T;
  const long d = (long)H * 128, at = (long)vid * 128;
  const __nv_bfloat16* in = qkv + (long)tok * 3 * d + h * 128;
  __nv_bfloat16* out = dqkv + (long)tok * 3 * d + h * 128;
  float c[8], s[8];
  ld8(cosb + (long)t * 64 + 8 * l, c);
  ld8(sinb + (long)t * 64 + 8 * l, s);
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const Vec x = ldv(in + which * d, l);
    Vec g;
    if (which == 0 && dq_f32 != nullptr) {   // dQ straight from the attention kernel's fp32 accumulator
      ldf8(dq_f32 + at + 8 * l, g.lo);
      ldf8(dq_f32 + at + 64 + 8 * l, g.hi);
    } else {
      const __nv_bfloat16* gp = (which == 0 ? dq : dk) + at;
      ld8(gp + 8 * l, g.lo);
      if (which == 1 && key_offset) {
        // the upper half computed here was consumed by the next token (and by token 0 itself)
#pragma unroll
        for (int i = 0; i < 8; ++i) g.hi[i] = 0.f;
        if (t + 1 < T) ld8(gp + d + 64 + 8 * l, g.hi);
        if (t == 0) {
          float own[8];
          ld8(gp + 64 + 8 * l, own);
#pragma unroll
          for (int i = 0; i < 8; ++i) g.hi[i] += own[i];
        }
      } else {
        ld8(gp + 64 + 8 * l, g.hi);
      }
    }
    Vec o;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o.lo[i] = x.lo[i] * c[i] + x.hi[i] * s[i];
      o.hi[i] = -x.lo[i] * s[i] + x.hi[i] * c[i];
    }
    const float r = rsqrtf(dot_pairs(o, o) * (1.f / 128.f) + eps);
    const float k = r * r * r * dot_pairs(o, g) * (1.f / 128.f);
    Vec w;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float d1 = r * g.lo[i] - k * o.lo[i], d2 = r * g.hi[i] - k * o.hi[i];
      w.lo[i] = d1 * c[i] - d2 * s[i];
      w.hi[i] = d1 * s[i] + d2 * c[i];
    }
    if (valid) stv(out + which * d, l, w);
  }
  Vec g = ldv(dv + at, l);
  if (dv_extra != nullptr) {    // second consumer of v (exclusive self-attention)
    const Vec x = ldv(dv_extra + at, l);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      g.lo[i] += x.lo[i];
      g.hi[i] += x.hi[i];
    }
  }
  if (valid) stv(out + 2 * d, l, g);
  if (ve != nullptr) {
    const float gt = gate[vid];
    const Vec e = ldv(ve + (long)tok * d + h * 128, l);
    const float dg = dot_quads(g, e);
    if (valid) {
      if (l == 0) dgate[vid] = dg;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        g.lo[i] *= gt;
        g.hi[i] *= gt;
      }
      stv(dve + (long)tok * d + h * 128, l, g);
    }
  }
}

// ---------------------------------------------------------------------------------------------- after attention
// alpha: fp32 [H] (raw, tanh applied here) or null = no exclusive self-attention.
__global__ void __launch_bounds__(kThreads)
attn_post_fwd_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ v, const float* __restrict__ gate,
                     const float* __restrict__ alpha, __nv_bfloat16* __restrict__ out, unsigned n, unsigned H, float xsa_eps) {
  const int l = threadIdx.x & 7;
  const unsigned steps = (n + gridDim.x * kVecPerBlock - 1) / (gridDim.x * kVecPerBlock);
  for (unsigned it = 0; it < steps; ++it) {
    const unsigned id = (it * gridDim.x + blockIdx.x) * kVecPerBlock + (threadIdx.x >> 3);
    const bool valid = id < n;
    const unsigned vid = valid ? id : n - 1;
    const long at = (long)vid * 128;
    Vec yy = ldv(y + at, l);
    const float s = gate[vid];
    if (alpha != nullptr) {
      const Vec vv = ldv(v + at, l);
      const float nn = fmaxf(sqrtf(dot_quads(vv, vv)), xsa_eps);
      const float c = dot_quads(yy, vv) / nn;
      const float k = tanhf(alpha[vid % H]) * c / nn;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        yy.lo[i] -= k * vv.lo[i];
        yy.hi[i] -= k * vv.hi[i];
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      yy.lo[i] *= s;
      yy.hi[i] *= s;
    }
    if (valid) stv(out + at, l, yy);
  }
}

// g: gradient of the gated output. Writes dy (gradient of the attention output), dgate (w.r.t. the gate value),
// delta[b, h, t] = sum_d dy * y, and with alpha: dv_x (this op's gradient of v) and dalpha[H] += (atomics, one per
// block and head).
__global__ void __launch_bounds__(kThreads)
attn_post_bwd_kernel(const __nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ v,
                     const float* __restrict__ gate, const float* __restrict__ alpha, __nv_bfloat16* __restrict__ dy,
                     float* __restrict__ dgate, float* __restrict__ delta, __nv_bfloat16* __restrict__ dv_x, float* __restrict__ dalpha,
                     unsigned n, unsigned H, unsigned T, float xsa_eps) {
  __shared__ float dal[64];
  const int l = threadIdx.x & 7;
  if (alpha != nullptr) {
    if (threadIdx.x < 64) dal[threadIdx.x] = 0.f;
    __syncthreads();
  }
  const unsigned steps = (n + gridDim.x * kVecPerBlock - 1) / (gridDim.x * kVecPerBlock);
  for (unsigned it = 0; it < steps; ++it) {
    const unsigned id = (it * gridDim.x + blockIdx.x) * kVecPerBlock + (threadIdx.x >> 3);
    const bool valid = id < n;
    const unsigned vid = valid ? id : n - 1;
    const unsigned tok = vid / H, h = vid - tok * H;
    const long at = (long)vid * 128;
    const Vec gg = ldv(g + at, l), yy = ldv(y + at, l);
    const float s = gate[vid];
    Vec d;       // gradient of the attention output
    float dg;    // sum_d g * (output before the gate)
    if (alpha != nullptr) {
      const Vec vv = ldv(v + at, l);
      const float nrm = sqrtf(dot_quads(vv, vv));
      const float inv = 1.f / fmaxf(nrm, xsa_eps);
      const float c = dot_quads(yy, vv) * inv;                // y . u,  u = v / max(|v|, eps)
      const float a = tanhf(alpha[h]);
      const float gy = dot_quads(gg, yy), gu = dot_quads(gg, vv) * inv;
      dg = gy - a * c * gu;                                   // g . (y - a c u)
      const float p = s * gu;                                 // (s g) . u
      Vec du;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float d0 = s * gg.lo[i], d1 = s * gg.hi[i];
        d.lo[i] = d0 - a * p * (vv.lo[i] * inv);
        d.hi[i] = d1 - a * p * (vv.hi[i] * inv);
        du.lo[i] = -a * (p * yy.lo[i] + c * d0);
        du.hi[i] = -a * (p * yy.hi[i] + c * d1);
      }
      // v -> u = v / max(|v|, eps): the projection term only where the norm is not clamped
      const float proj = dot_quads(du, vv) * inv;
      const float duu = nrm > xsa_eps ? proj : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        du.lo[i] = (du.lo[i] - duu * vv.lo[i] * inv) * inv;
        du.hi[i] = (du.hi[i] - duu * vv.hi[i] * inv) * inv;
      }
      if (valid) {
        stv(dv_x + at, l, du);
        if (l == 0) atomicAdd(&dal[h], -c * p * (1.f - a * a));
      }
    } else {
      dg = dot_quads(gg, yy);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        d.lo[i] = s * gg.lo[i];
        d.hi[i] = s * gg.hi[i];
      }
    }
    const float dl = dot_quads(d, yy);
    if (valid) {
      if (l == 0) {
        dgate[vid] = dg;
        delta[((long)(tok / T) * H + h) * T + tok % T] = dl;
      }
      stv(dy + at, l, d);
    }
  }
  if (alpha != nullptr) {
    __syncthreads();
    if (threadIdx.x < H && dal[threadIdx.x] != 0.f) atomicAdd(dalpha + threadIdx.x, dal[threadIdx.x]);
  }
}

// ---------------------------------------------------------------------------------------------- IHA weight mixing
// W, out: [P, H, J] bf16 (J = head_dim * d_in); mix: [P, H, H] fp32, used rounded to bf16 as the reference's autocast
// matmul does. One thread per pair of columns.
template <int H>
__global__ void iha_mix_fwd_kernel(const float* __restrict__ mix, const __nv_bfloat16* __restrict__ W,
                                   __nv_bfloat16* __restrict__ out, long J) {
  __shared__ float sm[H * H];
  const int p = blockIdx.y;
  for (int i = threadIdx.x; i < H * H; i += blockDim.x)
    sm[i] = __bfloat162float(__float2bfloat16(mix[(long)p * H * H + i]));
  __syncthreads();
  const long j = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 2;
  if (j >= J) return;
  const __nv_bfloat16* w = W + (long)p * H * J + j;
  float2 x[H];
#pragma unroll
  for (int m = 0; m < H; ++m) x[m] = ld2(w + (long)m * J);
  __nv_bfloat16* o = out + (long)p * H * J + j;
#pragma unroll
  for (int h = 0; h < H; ++h) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int m = 0; m < H; ++m) {
      a += sm[h * H + m] * x[m].x;
      b += sm[h * H + m] * x[m].y;
    }
    st2(o + (long)h * J, a, b);
  }
}

// gradW[p, m, j] += sum_h mix[p, h, m] * dWp[p, h, j]      (fp32 accumulate into the gradient arena)
template <int H>
__global__ void iha_mix_bwd_w_kernel(const float* __restrict__ mix, const __nv_bfloat16* __restrict__ dWp,
                                     float* __restrict__ gradW, long J) {
  __shared__ float sm[H * H];
  const int p = blockIdx.y;
  for (int i = threadIdx.x; i < H * H; i += blockDim.x)
    sm[i] = __bfloat162float(__float2bfloat16(mix[(long)p * H * H + i]));
  __syncthreads();
  const long j = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 2;
  if (j >= J) return;
  const __nv_bfloat16* g = dWp + (long)p * H * J + j;
  float2 x[H];
#pragma unroll
  for (int h = 0; h < H; ++h) x[h] = ld2(g + (long)h * J);
  float* o = gradW + (long)p * H * J + j;
#pragma unroll
  for (int m = 0; m < H; ++m) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int h = 0; h < H; ++h) {
      a += sm[h * H + m] * x[h].x;
      b += sm[h * H + m] * x[h].y;
    }
    // fire-and-forget vector reduction: a load-add-store here would serialise H DRAM round trips per thread
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(o + (long)m * J), "f"(a), "f"(b) : "memory");
  }
}

// dmix[p, h, m] += sum_j dWp[p, h, j] * W[p, m, j].  Each CTA stages `kCols` columns of both operands in shared memory
// (rows padded by one word against bank conflicts). The H x H result is cut into 4 x 4 register blocks; a thread owns
// one block for one slice of the staged columns, so every shared-memory word it loads feeds four multiply-adds.
// Slices are combined with shared-memory atomics, CTAs with one global atomicAdd per entry.
constexpr int kCols = 512;
constexpr int kChunksPerCta = 3;
template <int H>
__global__ void __launch_bounds__(kThreads)
iha_mix_bwd_mix_kernel(const __nv_bfloat16* __restrict__ dWp, const __nv_bfloat16* __restrict__ W,
                       float* __restrict__ dmix, long J) {
  constexpr int kStride = kCols + 2;
  constexpr int HB = (H + 3) / 4;                 // 4-row blocks per side
  constexpr int HP = HB * 4;                      // padded head count (extra rows are zero)
  constexpr int kBlocks = HB * HB;
  constexpr int kSlices = kThreads / kBlocks > 0 ? kThreads / kBlocks : 1;
  constexpr int kSliceCols = (kCols / 2 + kSlices - 1) / kSlices;   // bf16 pairs per slice
  __shared__ __nv_bfloat16 sg[HP * kStride];
  __shared__ __nv_bfloat16 sw[HP * kStride];
  __shared__ float sacc[HP * HP];
  const int p = blockIdx.y;
  for (int i = threadIdx.x; i < HP * HP; i += kThreads) sacc[i] = 0.f;
  const int blk = threadIdx.x % kBlocks, slice = threadIdx.x / kBlocks;
  const int bh = (blk / HB) * 4, bm = (blk % HB) * 4;
  const bool active = slice < kSlices;
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
  for (int ch = 0; ch < kChunksPerCta; ++ch) {
    const long j0 = ((long)blockIdx.x * kChunksPerCta + ch) * kCols;
    if (j0 >= J) break;
    const int ncols = (int)min((long)kCols, J - j0);
    __syncthreads();
    for (int i = threadIdx.x; i < HP * (kCols / 2); i += kThreads) {
      const int row = i / (kCols / 2), c2 = (i - row * (kCols / 2)) * 2;
      __nv_bfloat162 a = __floats2bfloat162_rn(0.f, 0.f), b = a;
      if (row < H && c2 < ncols) {
        a = *reinterpret_cast<const __nv_bfloat162*>(dWp + ((long)p * H + row) * J + j0 + c2);
        b = *reinterpret_cast<const __nv_bfloat162*>(W + ((long)p * H + row) * J + j0 + c2);
      }
      *reinterpret_cast<__nv_bfloat162*>(sg + row * kStride + c2) = a;
      *reinterpret_cast<__nv_bfloat162*>(sw + row * kStride + c2) = b;
    }
    __syncthreads();
    if (active) {
      const int c_lo = slice * kSliceCols, c_hi = min(kCols / 2, c_lo + kSliceCols);
      for (int c = c_lo; c < c_hi; ++c) {
        float2 g[4], w[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          g[a] = ld2(sg + (bh + a) * kStride + 2 * c);
          w[a] = ld2(sw + (bm + a) * kStride + 2 * c);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[a][b] += g[a].x * w[b].x + g[a].y * w[b].y;
      }
    }
  }
  if (active) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) atomicAdd(&sacc[(bh + a) * HP + bm + b], acc[a][b]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < H * H; i += kThreads) {
    const int h = i / H, m = i - h * H;
    atomicAdd(dmix + (long)p * H * H + i, sacc[h * HP + m]);
  }
}


// ---------------------------------------------------------------------------------------------- per-head gates
// gate[r, h] = scale * sigmoid(bf16(sum_c a[r, c] * bf16(W[h, c]))) over the first nc channels of the normed input
// (the reference's attn_gate / ve_gate linears under bf16 autocast, train.py:296-312). One thread per (row, head).
__global__ void gate_fwd_kernel(const __nv_bfloat16* __restrict__ a, long lda, const float* __restrict__ W,
                                float* __restrict__ gate, long M, int H, int nc, float scale) {
  extern __shared__ float gsm[];   // [H * nc] weights rounded to bf16
  for (int i = threadIdx.x; i < H * nc; i += blockDim.x) gsm[i] = __bfloat162float(__float2bfloat16(W[i]));
  __syncthreads();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= M * H) return;
  const long r = idx / H;
  const int h = (int)(idx - r * H);
  const __nv_bfloat16* ar = a + r * lda;
  float z = 0.f;
  for (int c = 0; c < nc; ++c) z += __bfloat162float(ar[c]) * gsm[h * nc + c];
  z = __bfloat162float(__float2bfloat16(z));
  gate[idx] = scale / (1.f + __expf(-z));
}

// dz = dgate * gate * (1 - gate / scale);  dW[h, c] += sum_r dz[r, h] * a[r, c];  da[r, c] += bf16(sum_h dz[r, h] * bf16(W[h, c])).
// A CTA stages kGateRows rows; thread (h, c) owns one weight-gradient entry, then the threads sweep the (row, c) pairs.
constexpr int kGateRows = 64;
__global__ void gate_bwd_kernel(const float* __restrict__ dgate, const float* __restrict__ gate,
                                const __nv_bfloat16* __restrict__ a, long lda, const float* __restrict__ W,
                                float* __restrict__ dW, __nv_bfloat16* __restrict__ da, long ldda, long M, int H, int nc,
                                float scale) {
  extern __shared__ float gsm[];
  float* sw = gsm;                       // [H * nc]
  float* sdz = sw + H * nc;              // [kGateRows * H]
  float* sa = sdz + kGateRows * H;       // [kGateRows * nc]
  const long r0 = (long)blockIdx.x * kGateRows;
  const int rows = (int)min((long)kGateRows, M - r0);
  for (int i = threadIdx.x; i < H * nc; i += blockDim.x) sw[i] = __bfloat162float(__float2bfloat16(W[i]));
  for (int i = threadIdx.x; i < rows * H; i += blockDim.x) {
    const float g = gate[r0 * H + i];
    sdz[i] = dgate[r0 * H + i] * g * (1.f - g / scale);
  }
  for (int i = threadIdx.x; i < rows * nc; i += blockDim.x) {
    const int r = i / nc, c = i - r * nc;
    sa[i] = __bfloat162float(a[(r0 + r) * lda + c]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < H * nc; e += blockDim.x) {
    const int h = e / nc, c = e - h * nc;
    float acc = 0.f;
    for (int r = 0; r < rows; ++r) acc += sdz[r * H + h] * sa[r * nc + c];
    atomicAdd(dW + e, acc);
  }
  for (int i = threadIdx.x; i < rows * nc; i += blockDim.x) {
    const int r = i / nc, c = i - r * nc;
    float acc = 0.f;
    for (int h = 0; h < H; ++h) acc += sdz[r * H + h] * sw[h * nc + c];
    __nv_bfloat16* d = da + (r0 + r) * ldda + c;
    *d = __float2bfloat16(__bfloat162float(*d) + __bfloat162float(__float2bfloat16(acc)));
  }
}

inline int rc() { return cudaGetLastError() == cudaSuccess ? 0 : -5; }

// The per-head vector kernels count vectors in 32 bits and use 16-byte accesses.
inline bool vectors_ok(long n, std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return false;
  return n <= 0x7fffffffL - kThreads;
}

constexpr int kIhaMaxHeads = 32;     // 2 x 32 registers of columns per thread
constexpr int kIhaMaxDmixHeads = 20; // staging of iha_mix_bwd_mix_kernel in 48 KB of static shared memory

template <int H>
int iha_launch(int which, const float* mix, const void* W, const void* dWp, void* out, float* gradW, float* dmix, int P,
               long J, cudaStream_t s) {
  const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(W);
  const __nv_bfloat16* g = reinterpret_cast<const __nv_bfloat16*>(dWp);
  const dim3 grid((unsigned)((J / 2 + kThreads - 1) / kThreads), P);
  if (which == 0) {
    iha_mix_fwd_kernel<H><<<grid, kThreads, 0, s>>>(mix, w, reinterpret_cast<__nv_bfloat16*>(out), J);
  } else {
    if (H > kIhaMaxDmixHeads && dmix != nullptr) return -7;
    iha_mix_bwd_w_kernel<H><<<grid, kThreads, 0, s>>>(mix, g, gradW, J);
    if constexpr (H <= kIhaMaxDmixHeads) if (dmix != nullptr) {   // callers with a split-K GEMM at hand form dmix = dW' W^T there and pass null
      const long chunks = (J + kCols - 1) / kCols;
      const dim3 grid2((unsigned)((chunks + kChunksPerCta - 1) / kChunksPerCta), P);
      iha_mix_bwd_mix_kernel<H><<<grid2, kThreads, 0, s>>>(g, w, dmix, J);
    }
  }
  return rc();
}

template <int H>
int iha_select(int which, int heads, const float* mix, const void* W, const void* dWp, void* out, float* gradW, float* dmix,
               int P, long J, cudaStream_t s) {
  if (heads == H) return iha_launch<H>(which, mix, W, dWp, out, gradW, dmix, P, J, s);
  if constexpr (H > 1) return iha_select<H - 1>(which, heads, mix, W, dWp, out, gradW, dmix, P, J, s);
  return -7;  // unsupported head count: the caller falls back to library matmuls
}

int iha_dispatch(int which, int H, const float* mix, const void* W, const void* dWp, void* out, float* gradW,
                 float* dmix, int P, long J, cudaStream_t s) {
  if (J % 2) return -2;
  // The columns of all heads sit in registers, so the head count is a template parameter; every count up to kIhaMaxHeads
  // has an instance. A head count without one goes to library matmuls, for which a [5, 5] x [5, 81920] product is a bad
  // shape: with 5 heads of d = 640 the backward of one layer took 1450 us there and takes about 15 us here.
  return iha_select<kIhaMaxHeads>(which, H, mix, W, dWp, out, gradW, dmix, P, J, s);
}

}  // namespace

#define BF(p) reinterpret_cast<const __nv_bfloat16*>(p)
#define BFM(p) reinterpret_cast<__nv_bfloat16*>(p)

// qkv: [tokens, 3*H*128]; ve: [tokens, H*128] or null; gate: fp32 [tokens, H] (only read when ve != null)
extern "C" int sr_qkv_prep_fwd(const void* qkv, const void* ve, const float* gate, const void* cosb, const void* sinb,
                               void* q, void* k, void* v, long tokens, int H, int T, float eps, int key_offset,
                               cudaStream_t s) {
  const long n = tokens * H;
  if (n <= 0) return 0;
  if (!vectors_ok(n, {qkv, ve, cosb, sinb, q, k, v})) return -2;
  qkv_prep_fwd_kernel<<<(unsigned)((n + kVecPerBlock - 1) / kVecPerBlock), kThreads, 0, s>>>(
      BF(qkv), BF(ve), gate, BF(cosb), BF(sinb), BFM(q), BFM(k), BFM(v), n, H, T, eps, key_offset);
  return rc();
}
extern "C" int sr_qkv_prep_bwd(const void* qkv, const void* ve, const float* gate, const void* cosb, const void* sinb,
                               const void* dq, const void* dk, const void* dv, void* dqkv, void* dve, float* dgate,
                               long tokens, int H, int T, float eps, int key_offset, const void* dv_extra,
                               cudaStream_t s) {
  const long n = tokens * H;
  if (n <= 0) return 0;
  if (!vectors_ok(n, {qkv, ve, cosb, sinb, dq, dk, dv, dqkv, dve, dv_extra})) return -2;
  qkv_prep_bwd_kernel<<<(unsigned)((n + kVecPerBlock - 1) / kVecPerBlock), kThreads, 0, s>>>(
      BF(qkv), BF(ve), gate, BF(cosb), BF(sinb), BF(dq), BF(dk), BF(dv), BFM(dqkv), BFM(dve), dgate, n, H, T, eps,
      nullptr, key_offset, BF(dv_extra));
  return rc();
}
// Same with dQ given as the fp32 accumulator of the attention backward, (tokens, H, 128) contiguous.
extern "C" int sr_qkv_prep_bwd_f32dq(const void* qkv, const void* ve, const float* gate, const void* cosb,
                                     const void* sinb, const float* dq_f32, const void* dk, const void* dv, void* dqkv,
                                     void* dve, float* dgate, long tokens, int H, int T, float eps, int key_offset,
                                     const void* dv_extra, cudaStream_t s) {
  const long n = tokens * H;
  if (n <= 0) return 0;
  if (!vectors_ok(n, {qkv, ve, cosb, sinb, dq_f32, dk, dv, dqkv, dve, dv_extra})) return -2;
  qkv_prep_bwd_kernel<<<(unsigned)((n + kVecPerBlock - 1) / kVecPerBlock), kThreads, 0, s>>>(
      BF(qkv), BF(ve), gate, BF(cosb), BF(sinb), nullptr, BF(dk), BF(dv), BFM(dqkv), BFM(dve), dgate, n, H, T, eps,
      dq_f32, key_offset, BF(dv_extra));
  return rc();
}

// y, v, out: [tokens, H, 128] bf16 contiguous; gate: fp32 [tokens, H]; alpha: fp32 [H] or null (v is then unused).
extern "C" int sr_attn_post_fwd(const void* y, const void* v, const float* gate, const float* alpha, void* out, long tokens,
                                int H, float xsa_eps, cudaStream_t s) {
  const long n = tokens * H;
  if (n <= 0) return 0;
  if (H > 64 || !vectors_ok(n, {y, alpha != nullptr ? v : nullptr, out})) return -2;
  long blocks = (n + kVecPerBlock - 1) / kVecPerBlock;
  const long cap = (long)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  attn_post_fwd_kernel<<<(unsigned)blocks, kThreads, 0, s>>>(BF(y), BF(v), gate, alpha, BFM(out), n, H, xsa_eps);
  return rc();
}
// g: gradient of `out`. dy, dv_x: [tokens, H, 128] bf16; dgate: fp32 [tokens, H]; delta: fp32 [B, H, T] with tokens = B * T;
// dalpha: fp32 [H], ADDED to (the caller passes the parameter's gradient buffer). dv_x / dalpha only with alpha.
extern "C" int sr_attn_post_bwd(const void* g, const void* y, const void* v, const float* gate, const float* alpha, void* dy,
                                float* dgate, float* delta, void* dv_x, float* dalpha, long tokens, int H, int T,
                                float xsa_eps, cudaStream_t s) {
  const long n = tokens * H;
  if (n <= 0) return 0;
  if (H > 64 || (alpha != nullptr && (dv_x == nullptr || dalpha == nullptr))) return -2;
  if (!vectors_ok(n, {g, y, alpha != nullptr ? v : nullptr, dy, alpha != nullptr ? dv_x : nullptr})) return -2;
  long blocks = (n + kVecPerBlock - 1) / kVecPerBlock;
  const long cap = (long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  attn_post_bwd_kernel<<<(unsigned)blocks, kThreads, 0, s>>>(BF(g), BF(y), BF(v), gate, alpha, BFM(dy), dgate, delta,
                                                             BFM(dv_x), dalpha, n, H, T, xsa_eps);
  return rc();
}
// out[p] = bf16(mix[p]) @ W[p] for P stacked projections, W viewed as [P, H, J]
extern "C" int sr_iha_mix_fwd(const float* mix, const void* W, void* out, int P, int H, long J, cudaStream_t s) {
  return iha_dispatch(0, H, mix, W, nullptr, out, nullptr, nullptr, P, J, s);
}
// gradW[p] += bf16(mix[p])^T @ dWp[p] (fp32) and dmix[p] += dWp[p] @ W[p]^T (fp32, atomically accumulated)
extern "C" int sr_iha_mix_bwd(const float* mix, const void* W, const void* dWp, float* gradW, float* dmix, int P, int H,
                              long J, cudaStream_t s) {
  return iha_dispatch(1, H, mix, W, dWp, nullptr, gradW, dmix, P, J, s);
}

// gate[M, H] (fp32) = scale * sigmoid(a[:, :nc] @ bf16(W)^T); a: bf16 rows with leading dimension lda; W: fp32 [H, nc]
extern "C" int sr_gate_fwd(const void* a, long lda, const float* W, float* gate, long M, int H, int nc, float scale,
                           cudaStream_t s) {
  if (M <= 0) return 0;
  const long n = M * H;
  gate_fwd_kernel<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, H * nc * sizeof(float), s>>>(BF(a), lda, W, gate,
                                                                                                     M, H, nc, scale);
  return rc();
}
// Backward of sr_gate_fwd: dW (fp32 [H, nc]) is accumulated into, da[:, :nc] (bf16, leading dimension ldda) is added to.
extern "C" int sr_gate_bwd(const float* dgate, const float* gate, const void* a, long lda, const float* W, float* dW,
                           void* da, long ldda, long M, int H, int nc, float scale, cudaStream_t s) {
  if (M <= 0) return 0;
  const size_t smem = (size_t)(H * nc + kGateRows * H + kGateRows * nc) * sizeof(float);
  if (smem > 48 * 1024) return -2;
  gate_bwd_kernel<<<(unsigned)((M + kGateRows - 1) / kGateRows), kThreads, smem, s>>>(dgate, gate, BF(a), lda, W, dW,
                                                                                     BFM(da), ldda, M, H, nc, scale);
  return rc();
}
