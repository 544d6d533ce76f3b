// Backward of the gated delta rule with one log-decay per head, chunk by chunk.
//
// The forward is the recurrence of gated_delta.cu. For the gradients a chunk of 64 tokens is a handful of dense 64-row
// products, and only the state has to travel from chunk to chunk. With G_t the running sum of the log-decays inside the
// chunk, S the state [Dk x Dv] entering it, E[t,j] = exp(G_t - G_j):
//     A[t,j] = beta_j (k_t . k_j) E[t,j]  (j < t)        P[t,j] = beta_j (q_t . k_j) E[t,j]  (j <= t)
//     R      = (I + A)^-1 (V - Kd S)                     Kd = exp(G) K,  Qd = exp(G) Q
//     O      = Qd S + P R
//     S_next = exp(G_C) S + Kend^T R                     Kend_j = beta_j exp(G_C - G_j) k_j
// Every exponential is of a non-positive number. With W = (I + A)^-1 Kd and U = (I + A)^-1 V, which need no state, the part
// that runs in sequence is R = U - W S and the state update: two small products per chunk, independent for every slice of
// value columns. The gradients have the same shape, last chunk first, with dS the gradient of the state leaving a chunk:
//     dRhs    = X + Y dS         X = (I + A)^-T P^T dO,  Y = (I + A)^-T Kend
//     dS_prev = exp(G_C) dS + Z - Kd^T dRhs,             Z = Qd^T dO                       dV = dRhs
// So there are three kernels: prep (all chunks at once), scan (in sequence, one CTA per head and 32 value columns; once
// forward for the states, once backward), and grads (all chunks at once). All arithmetic is fp32 FMA as in the recurrence;
// q, k, v may be bf16 or fp32. (The same chunks give the forward as well, in 890 us against the recurrence's 1650. That is not
// used: its other rounding travels through every later layer of a model.)
//
// What bounds it: shared-memory reads of the 64 x 64 x n products (a thread owns 4 x 4 results) and, for the scan, the
// latency of n_chunks dependent steps, which is why its operands are prefetched with cp.async.
// Measured, (B, T, H) = (4, 2048, 14), Dk = 64, Dv = 128: 2.0 ms (gradients through the PyTorch form: about 17 ms in 2900
// launches); prep 730, scan 240 each way, grads 815 us.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace {

constexpr int C = 64;          // tokens per chunk
constexpr int kThreads = 256;  // 16 x 16 threads; thread (ty, tx) owns rows ty + 16 i and columns tx + 16 j
constexpr int VS = 32;         // value columns per slice
constexpr int LC = C + 4;      // row stride (floats) of a 64-wide tile: 16-byte rows, 4-bank skew between rows
constexpr int LV = VS + 4;

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ void put(float* p, float x) { *p = x; }
__device__ __forceinline__ void put(__nv_bfloat16* p, float x) { *p = __float2bfloat16(x); }

// exp(x) to about one unit in the last place: x = n ln2 + r (ln2 in two parts, n * hi is exact), Taylor
// polynomial of e^r on |r| <= ln2 / 2 (the first term left out is 5e-9), exponent set by adding n to its bits. The ex2
// instruction alone is two units off, and every entry of A, P and their gradients carries one of these factors.
__device__ __forceinline__ float decay_exp(float x) {
  if (x < -87.f) return 0.f;                       // below the smallest normal number
  if (x > 88.f) return __int_as_float(0x7f800000); // a growing state: not what the layers do, but not refused either
  const float n = rintf(x * 1.44269504f);
  const float r = fmaf(-n, 1.42860682e-6f, fmaf(-n, 0.693145752f, x));
  float p = 1.f / 5040.f;
  p = fmaf(p, r, 1.f / 720.f);
  p = fmaf(p, r, 1.f / 120.f);
  p = fmaf(p, r, 1.f / 24.f);
  p = fmaf(p, r, 1.f / 6.f);
  p = fmaf(p, r, 0.5f);
  p = fmaf(p, r, 1.f);
  p = fmaf(p, r, 1.f);
  return __int_as_float(__float_as_int(p) + (static_cast<int>(n) << 23));
}

// acc[i][j] += sum_k A(ty + 16 i, k) B(k, tx + 16 j). A_KC: A stored [row][k] (else [k][row]); B_KC: B stored [col][k]
// (else [k][col]).
template <int NI, int NJ, int K, bool A_KC, bool B_KC>
__device__ __forceinline__ void mm(float (&acc)[NI][NJ], const float* A, int lda, const float* B, int ldb) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float a[NI][4], b[NJ][4];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      if (A_KC) {
        const float4 t = *reinterpret_cast<const float4*>(A + (ty + 16 * i) * lda + k);
        a[i][0] = t.x; a[i][1] = t.y; a[i][2] = t.z; a[i][3] = t.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) a[i][e] = A[(k + e) * lda + ty + 16 * i];
      }
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      if (B_KC) {
        const float4 t = *reinterpret_cast<const float4*>(B + (tx + 16 * j) * ldb + k);
        b[j][0] = t.x; b[j][1] = t.y; b[j][2] = t.z; b[j][3] = t.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) b[j][e] = B[(k + e) * ldb + tx + 16 * j];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j] = fmaf(a[i][e], b[j][e], acc[i][j]);
  }
}
template <int NI, int NJ>
__device__ __forceinline__ void zero(float (&acc)[NI][NJ]) {
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j] = 0.f;
}
// f(row, col, value) for every result of this thread
template <int NI, int NJ, typename F>
__device__ __forceinline__ void each(float (&acc)[NI][NJ], F f) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) f(ty + 16 * i, tx + 16 * j, acc[i][j]);
}

struct Dims {
  int T, H, Dv, n;   // n = chunks per sequence
};
// token row of chunk-local token t, in units of rows of the [B, T, H, *] inputs
__device__ __forceinline__ long in_row(const Dims& d, int bh, int c, int t) {
  const int b = bh / d.H, h = bh - b * d.H;
  return ((long)b * d.T + (long)c * C + t) * d.H + h;
}

// rows of the chunk into shared memory (zero past the end of the sequence and past `width` valid columns)
template <int N, typename T>
__device__ __forceinline__ void load_rows(float* dst, int ld, const T* src, int row_len, int col0, int width, const Dims& d, int bh, int c) {
  for (int i = threadIdx.x; i < C * N; i += kThreads) {
    const int t = i / N, x = i - t * N;
    const bool ok = c * C + t < d.T && x < width;
    dst[t * ld + x] = ok ? to_f(src[in_row(d, bh, c, t) * row_len + col0 + x]) : 0.f;
  }
}
// running log-decay and beta of the chunk; tokens past the end decay by nothing and write nothing. 64 threads.
__device__ __forceinline__ void load_gates(float* G, float* beta, const float* g, const float* b, const Dims& d, int bh, int c) {
  const int t = threadIdx.x;
  if (t < C) {
    const bool ok = c * C + t < d.T;
    const long r = ok ? in_row(d, bh, c, t) : 0;
    G[t] = ok ? g[r] : 0.f;
    beta[t] = ok ? b[r] : 0.f;
  }
  __syncthreads();
  if (t < 32) {   // inclusive scan of 64 values by one warp
    float x0 = G[2 * t], x1 = x0 + G[2 * t + 1], s = x1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, s, o);
      if (t >= o) s += y;
    }
    const float before = s - x1;
    __syncwarp();
    G[2 * t] = before + x0;
    G[2 * t + 1] = s;
  }
  __syncthreads();
}

// X = (I + A)^-1 for the strictly lower triangular A [64][LC], 16 rows at a time: the rows above enter as a product, the
// 16 rows of the block are substituted by one thread per column.
__device__ __forceinline__ void invert_unit_lower(const float* A, float* X) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 1
  for (int blk = 0; blk < 4; ++blk) {
    const int r0 = blk * 16;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < r0; ++k) {
      const float a = A[(r0 + ty) * LC + k];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = fmaf(a, X[k * LC + tx + 16 * j], acc[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) X[(r0 + ty) * LC + tx + 16 * j] = (r0 + ty == tx + 16 * j ? 1.f : 0.f) - acc[j];
    __syncthreads();
    if (threadIdx.x < C) {
      const int col = threadIdx.x;
      float x[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        float s = X[(r0 + t) * LC + col];
#pragma unroll
        for (int k = 0; k < t; ++k) s = fmaf(-A[(r0 + t) * LC + r0 + k], x[k], s);
        x[t] = s;
        X[(r0 + t) * LC + col] = s;
      }
    }
    __syncthreads();
  }
}

// Scratch: rows are padded to whole chunks (row cc * 64 + t with cc = bh * n + c) and value columns to whole slices (DvP).
//   W [64 x Dk] = -(I + A)^-1 Kd       U [64 x DvP] = (I + A)^-1 V, overwritten by R       Ke [64 x Dk] = Kend
//   S [Dk x DvP] state entering the chunk        dec = exp(G_C)
//   Y [64 x Dk] = (I + A)^-T Kend      X [64 x DvP] = (I + A)^-T P^T dO, overwritten by dRhs     Kn [64 x Dk] = -Kd
//   Z [Dk x DvP] = Qd^T dO             dS [Dk x DvP] gradient of the state leaving the chunk
struct Scratch {
  float *W, *U, *Ke, *S, *dec, *Y, *X, *Kn, *Z, *dS;
};

template <int Dk>
constexpr int prep_smem() { return (2 * C * (Dk + 4) + 3 * C * LC + C * LV + 2 * C) * 4; }

template <int Dk, typename T>
__global__ void __launch_bounds__(kThreads)
gdn_prep_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const float* __restrict__ g,
                const float* __restrict__ beta, const T* __restrict__ dO, Scratch s, Dims d) {
  extern __shared__ __align__(16) float sm[];
  constexpr int LK = Dk + 4, NK = Dk / 16;
  float* sK = sm;
  float* sQ = sK + C * LK;
  float* sA = sQ + C * LK;
  float* sP = sA + C * LC;
  float* sT = sP + C * LC;
  float* sV = sT + C * LC;      // 64 x 32 slices of v, then of dO
  float* G = sV + C * LV;
  float* bt = G + C;
  const int c = blockIdx.x, bh = blockIdx.y;
  const long cc = (long)bh * d.n + c;
  load_rows<Dk>(sK, LK, k, Dk, 0, Dk, d, bh, c);
  load_rows<Dk>(sQ, LK, q, Dk, 0, Dk, d, bh, c);
  load_gates(G, bt, g, beta, d, bh, c);
  const float Gend = G[C - 1];
  {
    float acc[4][4];
    zero(acc);
    mm<4, 4, Dk, true, true>(acc, sK, LK, sK, LK);
    each(acc, [&](int t, int j, float x) { sA[t * LC + j] = j < t ? x * bt[j] * decay_exp(G[t] - G[j]) : 0.f; });
    zero(acc);
    mm<4, 4, Dk, true, true>(acc, sQ, LK, sK, LK);
    each(acc, [&](int t, int j, float x) {
      const float y = j <= t ? x * bt[j] * decay_exp(G[t] - G[j]) : 0.f;
      sP[t * LC + j] = y;
    });
  }
  __syncthreads();
  invert_unit_lower(sA, sT);
  // K -> Kend, Q -> Qd in place
  for (int i = threadIdx.x; i < C * Dk; i += kThreads) {
    const int t = i / Dk, x = i - t * Dk;
    const float kk = sK[t * LK + x], e = decay_exp(G[t]), ke = kk * bt[t] * decay_exp(Gend - G[t]);
    s.Ke[(cc * C + t) * Dk + x] = ke;
    s.Kn[(cc * C + t) * Dk + x] = -kk * e;
    sQ[t * LK + x] *= e;
    sK[t * LK + x] = ke;
  }
  if (threadIdx.x == 0) s.dec[cc] = decay_exp(Gend);
  __syncthreads();
  {
    float acc[4][NK];
    zero(acc);
    mm<4, NK, C, false, false>(acc, sT, LC, sK, LK);       // Y = (I + A)^-T Kend
    each(acc, [&](int t, int x, float y) { s.Y[(cc * C + t) * Dk + x] = y; });
    float mx[4][4];
    zero(mx);
    mm<4, 4, C, false, true>(mx, sT, LC, sP, LC);          // (I + A)^-T P^T, over A
    each(mx, [&](int t, int j, float y) { sA[t * LC + j] = y; });
    __syncthreads();
    for (int i = threadIdx.x; i < C * Dk; i += kThreads) {
      const int t = i / Dk, x = i - t * Dk;
      const bool ok = c * C + t < d.T;
      sK[t * LK + x] = ok ? to_f(k[in_row(d, bh, c, t) * Dk + x]) * decay_exp(G[t]) : 0.f;
    }
    __syncthreads();
  }
  {
    float acc[4][NK];
    zero(acc);
    mm<4, NK, C, true, false>(acc, sT, LC, sK, LK);
    each(acc, [&](int t, int x, float y) { s.W[(cc * C + t) * Dk + x] = -y; });
  }
  const int DvP = (d.Dv + VS - 1) / VS * VS;
  for (int v0 = 0; v0 < d.Dv; v0 += VS) {
    float acc[4][2];
    __syncthreads();
    load_rows<VS>(sV, LV, v, d.Dv, v0, d.Dv - v0, d, bh, c);
    __syncthreads();
    zero(acc);
    mm<4, 2, C, true, false>(acc, sT, LC, sV, LV);
    each(acc, [&](int t, int x, float y) { s.U[(cc * C + t) * DvP + v0 + x] = y; });
    __syncthreads();
    load_rows<VS>(sV, LV, dO, d.Dv, v0, d.Dv - v0, d, bh, c);
    __syncthreads();
    zero(acc);
    mm<4, 2, C, true, false>(acc, sA, LC, sV, LV);
    each(acc, [&](int t, int x, float y) { s.X[(cc * C + t) * DvP + v0 + x] = y; });
    float az[NK][2];
    zero(az);
    mm<NK, 2, C, false, false>(az, sQ, LK, sV, LV);
    each(az, [&](int r, int x, float y) { s.Z[(cc * Dk + r) * DvP + v0 + x] = y; });
  }
}

// ---------------------------------------------------------------------------------------------- scan over chunks
__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// N columns (a multiple of 4) of `rows` rows
template <int N>
__device__ __forceinline__ void cp_tile(float* dst, int ld, const float* src, int row_len, int rows) {
  for (int i = threadIdx.x; i < rows * (N / 4); i += kThreads) {
    const int r = i / (N / 4), x = (i - r * (N / 4)) * 4;
    cp16(dst + r * ld + x, src + (long)r * row_len + x);
  }
}

template <int Dk>
constexpr int scan_smem() { return (2 * Dk * LV + 2 * (2 * C * (Dk + 4) + C * LV)) * 4; }

// State <- dec * State + Z + M2^T R with R = V + M1 State, chunk after chunk (REV: last first). V is overwritten by R and
// `saved` receives the state before each step. Forward: M1 = W, M2 = Kend, no Z. Backward: M1 = Y, M2 = -Kd.
template <int Dk, bool REV>
__global__ void __launch_bounds__(kThreads)
gdn_scan_kernel(const float* __restrict__ M1, const float* __restrict__ M2, float* __restrict__ V, const float* __restrict__ Z,
                const float* __restrict__ dec, float* __restrict__ saved, int n, int DvP) {
  extern __shared__ __align__(16) float sm[];
  constexpr int LK = Dk + 4, NK = Dk / 16, kBuf = 2 * C * LK + C * LV;
  float* St = sm;
  float* sZ = St + Dk * LV;
  float* buf = sZ + Dk * LV;
  const int bh = blockIdx.x, v0 = blockIdx.y * VS;
  auto fetch = [&](int step) {
    if (step < n) {
      const long cc = (long)bh * n + (REV ? n - 1 - step : step);
      float* t = buf + (step & 1) * kBuf;
      cp_tile<Dk>(t, LK, M1 + cc * C * Dk, Dk, C);
      cp_tile<Dk>(t + C * LK, LK, M2 + cc * C * Dk, Dk, C);
      cp_tile<VS>(t + 2 * C * LK, LV, V + cc * C * DvP + v0, DvP, C);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = threadIdx.x; i < Dk * LV; i += kThreads) St[i] = 0.f;
  fetch(0);
  for (int step = 0; step < n; ++step) {
    const long cc = (long)bh * n + (REV ? n - 1 - step : step);
    if (REV) {
      cp_tile<VS>(sZ, LV, Z + cc * Dk * DvP + v0, DvP, Dk);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    fetch(step + 1);      // its buffer was last read in the step before, which ended with a barrier
    if (REV) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else     asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float* t = buf + (step & 1) * kBuf;
    float* sV = const_cast<float*>(t) + 2 * C * LK;
    const float e = dec[cc];
    for (int i = threadIdx.x; i < Dk * VS; i += kThreads) {
      const int r = i / VS, x = i - r * VS;
      saved[(cc * Dk + r) * DvP + v0 + x] = St[r * LV + x];
    }
    float acc[4][2];
    zero(acc);
    mm<4, 2, Dk, true, false>(acc, t, LK, St, LV);
    each(acc, [&](int r, int x, float y) {
      const float z = sV[r * LV + x] + y;
      sV[r * LV + x] = z;
      V[(cc * C + r) * DvP + v0 + x] = z;
    });
    if (REV) asm volatile("cp.async.wait_group 1;" ::: "memory");   // Z; the operands of the next step stay in flight
    __syncthreads();
    float ns[NK][2];
    zero(ns);
    mm<NK, 2, C, false, false>(ns, t + C * LK, LK, sV, LV);
    each(ns, [&](int r, int x, float y) { St[r * LV + x] = e * St[r * LV + x] + y + (REV ? sZ[r * LV + x] : 0.f); });
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------- gradients
template <int Dk>
constexpr int grads_smem() {
  return (2 * C * (Dk + 4) + (2 * Dk * LV + 3 * C * LV > 2 * C * LC ? 2 * Dk * LV + 3 * C * LV : 2 * C * LC) + 4 * C + 8) * 4;
}
__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int Dk, typename T>
__global__ void __launch_bounds__(kThreads, Dk == 64 ? 2 : 1)
gdn_grads_kernel(const T* __restrict__ q, const T* __restrict__ k, const float* __restrict__ g, const float* __restrict__ beta,
                 const T* __restrict__ dO, Scratch s, T* __restrict__ dq, T* __restrict__ dk, T* __restrict__ dv,
                 float* __restrict__ dg, float* __restrict__ dbeta, Dims d) {
  extern __shared__ __align__(16) float sm[];
  constexpr int LK = Dk + 4, NK = Dk / 16;
  constexpr int kUnion = 2 * Dk * LV + 3 * C * LV > 2 * C * LC ? 2 * Dk * LV + 3 * C * LV : 2 * C * LC;
  float* sK = sm;
  float* sQ = sK + C * LK;
  float* sS = sQ + C * LK;         // value slices ...
  float* sdS = sS + Dk * LV;
  float* sO = sdS + Dk * LV;
  float* sR = sO + C * LV;
  float* sX = sR + C * LV;
  float* sM1 = sS;                 // ... later the two 64 x 64 matrices
  float* sM2 = sM1 + C * LC;
  float* G = sS + kUnion;
  float* bt = G + C;
  float* dG = bt + C;
  float* dB = dG + C;
  float* total = dB + C;
  const int c = blockIdx.x, bh = blockIdx.y;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const long cc = (long)bh * d.n + c;
  const int DvP = (d.Dv + VS - 1) / VS * VS;
  if (threadIdx.x < C) dG[threadIdx.x] = dB[threadIdx.x] = 0.f;
  if (threadIdx.x == 0) *total = 0.f;
  load_rows<Dk>(sK, LK, k, Dk, 0, Dk, d, bh, c);
  load_rows<Dk>(sQ, LK, q, Dk, 0, Dk, d, bh, c);
  load_gates(G, bt, g, beta, d, bh, c);
  const float Gend = G[C - 1];
  float aQ[4][NK], aK[4][NK], aP[4][4], aA[4][4];
  zero(aQ); zero(aK); zero(aP); zero(aA);
  float dend = 0.f;                // this thread's part of the gradient of G_C
  {
    float aE[4][NK];               // R dS^T
    zero(aE);
    for (int v0 = 0; v0 < d.Dv; v0 += VS) {
      __syncthreads();
      for (int i = threadIdx.x; i < Dk * VS; i += kThreads) {
        const int r = i / VS, x = i % VS;
        const float a = s.S[(cc * Dk + r) * DvP + v0 + x], b = s.dS[(cc * Dk + r) * DvP + v0 + x];
        sS[r * LV + x] = a;
        sdS[r * LV + x] = b;
        dend = fmaf(a, b, dend);
      }
      load_rows<VS>(sO, LV, dO, d.Dv, v0, d.Dv - v0, d, bh, c);
      for (int i = threadIdx.x; i < C * VS; i += kThreads) {
        const int t = i / VS, x = i % VS;
        sR[t * LV + x] = s.U[(cc * C + t) * DvP + v0 + x];
        const float y = s.X[(cc * C + t) * DvP + v0 + x];
        sX[t * LV + x] = y;
        if (c * C + t < d.T && v0 + x < d.Dv) put(dv + in_row(d, bh, c, t) * d.Dv + v0 + x, y);
      }
      __syncthreads();
      mm<4, NK, VS, true, true>(aQ, sO, LV, sS, LV);     // dQd
      mm<4, NK, VS, true, true>(aK, sX, LV, sS, LV);     // -dKd
      mm<4, NK, VS, true, true>(aE, sR, LV, sdS, LV);    // dKend
      mm<4, 4, VS, true, true>(aP, sO, LV, sR, LV);      // dP
      mm<4, 4, VS, true, true>(aA, sX, LV, sR, LV);      // -dA
    }
    dend *= decay_exp(Gend);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ty + 16 * i;
      const float e = decay_exp(G[t]), f0 = decay_exp(Gend - G[t]), f = bt[t] * f0;
      float rg = 0.f, re = 0.f;
#pragma unroll
      for (int j = 0; j < NK; ++j) {
        const float kk = sK[t * LK + tx + 16 * j], qq = sQ[t * LK + tx + 16 * j];
        aQ[i][j] *= e;
        const float kd = -aK[i][j] * e;
        rg += aQ[i][j] * qq + kd * kk;
        re += aE[i][j] * kk;
        aK[i][j] = kd + aE[i][j] * f;
      }
      rg = half_warp_sum(rg);
      re = half_warp_sum(re);
      if (tx == 0) {
        atomicAdd(&dG[t], rg - re * f);
        atomicAdd(&dB[t], re * f0);
        dend += re * f;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dend += __shfl_xor_sync(0xffffffffu, dend, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(total, dend);
  __syncthreads();                 // the slices have been read by everybody
  {
    float x1[4][4], x2[4][4];
    zero(x1); zero(x2);
    mm<4, 4, Dk, true, true>(x1, sQ, LK, sK, LK);
    mm<4, 4, Dk, true, true>(x2, sK, LK, sK, LK);
    float rows[4] = {0.f, 0.f, 0.f, 0.f}, cols[4] = {0.f, 0.f, 0.f, 0.f}, bcols[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = ty + 16 * i, u = tx + 16 * j;
        const float E = u <= t ? decay_exp(G[t] - G[u]) : 0.f;
        const float p = aP[i][j] * E, a = u < t ? -aA[i][j] * E : 0.f;
        const float y = p * x1[i][j] + a * x2[i][j];      // gradient of log E, before beta
        bcols[j] += y;
        rows[i] += y * bt[u];
        cols[j] += y * bt[u];
        sM1[t * LC + u] = p * bt[u];
        sM2[t * LC + u] = a * bt[u];
      }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float r = half_warp_sum(rows[i]);
      if (tx == 0) atomicAdd(&dG[ty + 16 * i], r);
      // the two rows of a warp share their columns
      const float cl = cols[i] + __shfl_xor_sync(0xffffffffu, cols[i], 16), b = bcols[i] + __shfl_xor_sync(0xffffffffu, bcols[i], 16);
      if ((threadIdx.x & 31) < 16) {
        atomicAdd(&dG[tx + 16 * i], -cl);
        atomicAdd(&dB[tx + 16 * i], b);
      }
    }
  }
  __syncthreads();
  mm<4, NK, C, true, false>(aQ, sM1, LC, sK, LK);
  mm<4, NK, C, false, false>(aK, sM1, LC, sQ, LK);
  mm<4, NK, C, true, false>(aK, sM2, LC, sK, LK);
  mm<4, NK, C, false, false>(aK, sM2, LC, sK, LK);
  each(aQ, [&](int t, int x, float y) { if (c * C + t < d.T) put(dq + in_row(d, bh, c, t) * Dk + x, y); });
  each(aK, [&](int t, int x, float y) { if (c * C + t < d.T) put(dk + in_row(d, bh, c, t) * Dk + x, y); });
  if (threadIdx.x < 32) {          // g_t enters G_t .. G_63: suffix sums
    const int l = threadIdx.x;
    const float x1 = dG[2 * l + 1] + (l == 31 ? *total : 0.f), x0 = dG[2 * l];
    float sum = x0 + x1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_down_sync(0xffffffffu, sum, o);
      if (l + o < 32) sum += y;
    }
    const float after = sum - (x0 + x1);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = 2 * l + e;
      if (c * C + t < d.T) {
        const long r = in_row(d, bh, c, t);
        dg[r] = e == 0 ? sum : after + x1;
        dbeta[r] = dB[t];
      }
    }
  }
}

struct Layout {
  long rk, rv, st, cs;   // floats of a [rows x Dk], [rows x DvP], [chunks x Dk x DvP], [chunks] array
  Layout(int B, int T, int H, int Dk, int Dv) {
    const long chunks = (long)B * H * ((T + C - 1) / C), DvP = (Dv + VS - 1) / VS * VS;
    rk = chunks * C * Dk;
    rv = chunks * C * DvP;
    st = chunks * Dk * DvP;
    cs = (chunks + 3) / 4 * 4;
  }
  long total() const { return 4 * rk + 2 * rv + 3 * st + cs; }
  Scratch split(float* p) const {
    auto take = [&](long n) { float* r = p; p += n; return r; };
    Scratch s{};
    s.W = take(rk); s.Ke = take(rk); s.U = take(rv); s.S = take(st); s.dec = take(cs);
    s.Y = take(rk); s.Kn = take(rk); s.X = take(rv); s.Z = take(st); s.dS = take(st);
    return s;
  }
};

template <typename K>
bool allow_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

template <int Dk, typename T>
int run_bwd(const T* q, const T* k, const T* v, const float* g, const float* beta, const T* dO, T* dq, T* dk, T* dv, float* dg, float* dbeta,
            float* scratch, int B, int T_, int H, int Dv, cudaStream_t st) {
  static const bool ok = allow_smem(gdn_prep_kernel<Dk, T>, prep_smem<Dk>()) && allow_smem(gdn_scan_kernel<Dk, false>, scan_smem<Dk>()) &&
                         allow_smem(gdn_scan_kernel<Dk, true>, scan_smem<Dk>()) && allow_smem(gdn_grads_kernel<Dk, T>, grads_smem<Dk>());
  if (!ok) return -4;
  const Layout l(B, T_, H, Dk, Dv);
  const Scratch s = l.split(scratch);
  const Dims d{T_, H, Dv, (T_ + C - 1) / C};
  const int slices = (Dv + VS - 1) / VS;
  const dim3 chunks(d.n, B * H), heads(B * H, slices);
  gdn_prep_kernel<Dk, T><<<chunks, kThreads, prep_smem<Dk>(), st>>>(q, k, v, g, beta, dO, s, d);
  gdn_scan_kernel<Dk, false><<<heads, kThreads, scan_smem<Dk>(), st>>>(s.W, s.Ke, s.U, nullptr, s.dec, s.S, d.n, slices * VS);
  gdn_scan_kernel<Dk, true><<<heads, kThreads, scan_smem<Dk>(), st>>>(s.Y, s.Kn, s.X, s.Z, s.dec, s.dS, d.n, slices * VS);
  gdn_grads_kernel<Dk, T><<<chunks, kThreads, grads_smem<Dk>(), st>>>(q, k, g, beta, dO, s, dq, dk, dv, dg, dbeta, d);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

int check(int B, int T, int H, int Dk, int Dv) {
  if ((Dk != 64 && Dk != 128) || Dv <= 0) return -2;
  if ((long)B * H > 65535) return -2;      // grid.y of the chunk kernels
  return 0;
}

}  // namespace

// Floats of scratch for one call (16-byte aligned buffer).
extern "C" long long sr_gdn_chunk_scratch(int B, int T, int H, int Dk, int Dv) {
  if (B <= 0 || T <= 0 || H <= 0 || Dk <= 0 || Dv <= 0) return 0;
  return Layout(B, T, H, Dk, Dv).total();
}

// Gradients of o = gated_delta_rule(q, k, v, g, beta) from dO. q, k, dq, dk: [B, T, H, Dk]; v, dv, dO: [B, T, H, Dv], all bf16 or
// (fp32 != 0) all fp32; g (log-decay), beta, dg, dbeta: fp32 [B, T, H]; all contiguous; Dk 64 or 128.
extern "C" int sr_gdn_chunk_bwd(const void* q, const void* k, const void* v, const float* g, const float* beta, const void* dO, void* dq,
                                void* dk, void* dv, float* dg, float* dbeta, float* scratch, int B, int T, int H, int Dk, int Dv, int fp32,
                                cudaStream_t s) {
  if (B <= 0 || T <= 0 || H <= 0) return 0;
  if (int rc = check(B, T, H, Dk, Dv)) return rc;
  using bf = __nv_bfloat16;
  if (fp32) {
    auto f = Dk == 64 ? run_bwd<64, float> : run_bwd<128, float>;
    return f((const float*)q, (const float*)k, (const float*)v, g, beta, (const float*)dO, (float*)dq, (float*)dk, (float*)dv, dg, dbeta,
             scratch, B, T, H, Dv, s);
  }
  auto f = Dk == 64 ? run_bwd<64, bf> : run_bwd<128, bf>;
  return f((const bf*)q, (const bf*)k, (const bf*)v, g, beta, (const bf*)dO, (bf*)dq, (bf*)dk, (bf*)dv, dg, dbeta, scratch, B, T, H, Dv, s);
}
