// Flash attention forward for sm_100a: causal with a left sliding window, head_dim 128, bf16, (B, T, H, D) layout.
//
// One CTA per (batch*head, 128-query tile). Warp roles (192 threads):
//   warp 0      TMA producer: Q once, then K_j / V_j tiles (128 keys) through a 2-stage ring
//   warp 1      MMA issuer + TMEM owner:  S_j = Q K_j^T   (SS, both operands K-major, accumulator in TMEM)
//                                          O  += P_j V_j   (SS, P from shared memory, V_j as an MN-major operand)
//   warps 2..5  softmax: thread i owns query row i (TMEM lane i), so row max / row sum need no shuffles. They read
//               S_j from TMEM, apply scale + mask, keep running (m, l), rescale O in TMEM when the max moved,
//               write P_j (bf16) into shared memory in the 128B-swizzled K-major layout, and at the end write
//               O / l and the log-sum-exp.
// S is double buffered in TMEM so S_{j+1} is computed while the softmax of tile j runs.
// Keys visible to query i: max(0, i - window) <= k <= i  (window < 0 means unlimited), the convention of
// flash_attn's window_size=(window, 0) that the reference uses (train.py:211-213, 432-438).
#include "sm100_common.cuh"

namespace {

using namespace sr;

constexpr int BQ = 128, D = 128;
constexpr int kThreads = 192;
constexpr uint32_t kQBytes = BQ * D * 2;           // 32 KB
constexpr uint32_t kQHalf = BQ * 128;              // one 64-column half of a 128-row tile: 128 rows x 128 B

// BKV = keys per tile. 128: one CTA per SM; 64: two CTAs per SM (their softmax and MMA phases overlap).
template <int BKV>
struct FwdCfg {
  static constexpr uint32_t kKVBytes = BKV * D * 2;       // K or V tile
  static constexpr uint32_t kKVHalf = BKV * 128;          // 64 d-columns of a K/V tile
  static constexpr uint32_t kPBytes = BQ * BKV * 2;
  static constexpr uint32_t kTmemCols = (BKV == 128) ? 512 : 256;   // 2 S buffers + O
  static constexpr int kSmemBytes = kQBytes + 4 * kKVBytes + kPBytes + 256;
};

struct FwdParams {
  __nv_bfloat16* out;   // [B, T, H, D]
  float* lse;           // [B, H, T]
  int B, T, H;
  int window;           // < 0: unlimited
  float scale_log2;     // softmax scale * log2(e)
  int* status;
};

template <int BKV>
__device__ __forceinline__ void kv_range(int q0, int T, int window, int& j_lo, int& j_hi) {
  const int q_last = min(q0 + BQ - 1, T - 1);
  j_hi = q_last / BKV;
  j_lo = (window < 0) ? 0 : max(0, q0 - window) / BKV;
}

template <int BKV>
__global__ void __launch_bounds__(kThreads, (BKV == 64) ? 2 : 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const FwdParams p) {
  using C_ = FwdCfg<BKV>;
  constexpr uint32_t kKVBytes = C_::kKVBytes, kKVHalf = C_::kKVHalf;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sK = smem + kQBytes;                       // 2 stages
  uint8_t* sV = sK + 2 * kKVBytes;                    // 2 stages
  uint8_t* sP = sV + 2 * kKVBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + C_::kPBytes);
  uint64_t* q_full = bars;            // 1
  uint64_t* k_full = bars + 1;        // 2
  uint64_t* v_full = bars + 3;        // 2
  uint64_t* kv_empty = bars + 5;      // 2
  uint64_t* s_full = bars + 7;        // 2
  uint64_t* p_full = bars + 9;        // 1 (count 128)
  uint64_t* pv_done = bars + 10;      // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_qt = (p.T + BQ - 1) / BQ;
  const int qt = n_qt - 1 - static_cast<int>(blockIdx.x);   // heavy (late) tiles first
  const int bh = blockIdx.y;
  const int b = bh / p.H, h = bh - b * p.H;
  const int q0 = qt * BQ;
  int j_lo, j_hi;
  kv_range<BKV>(q0, p.T, p.window, j_lo, j_hi);
  const int n_kv = j_hi - j_lo + 1;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&kv_empty[i], 1);
      mbar_init(&s_full[i], 1);
    }
    mbar_init(p_full, 128);
    mbar_init(pv_done, 1);
    *abort_flag = 0;
    if ((smem_u32(smem) & 1023u) != 0u) report_error(p.status, SR_ERR_BAD_ARG, 1000, 0);   // swizzle needs 1 KB alignment
    fence_barrier_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C_::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base;          // two buffers of BKV columns
  const uint32_t tmem_O = tmem_base + 2 * BKV;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_arrive_expect_tx(q_full, kQBytes);
      tma_load_4d(sQ, &map_q, q_full, 0, h, q0, b);
      tma_load_4d(sQ + kQHalf, &map_q, q_full, 64, h, q0, b);
      for (int it = 0; it < n_kv; ++it) {
        const int st = it & 1;
        const uint32_t ph = (it >> 1) & 1u;
        if (!mbar_wait(&kv_empty[st], ph ^ 1u, abort_flag, p.status, 1100)) break;
        const int k0 = (j_lo + it) * BKV;
        mbar_arrive_expect_tx(&k_full[st], kKVBytes);
        tma_load_4d(sK + st * kKVBytes, &map_k, &k_full[st], 0, h, k0, b);
        tma_load_4d(sK + st * kKVBytes + kKVHalf, &map_k, &k_full[st], 64, h, k0, b);
        mbar_arrive_expect_tx(&v_full[st], kKVBytes);
        tma_load_4d(sV + st * kKVBytes, &map_v, &v_full[st], 0, h, k0, b);
        tma_load_4d(sV + st * kKVBytes + kKVHalf, &map_v, &v_full[st], 64, h, k0, b);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc(1, 1, 0, 0, BQ, BKV);   // Q (K-major) x K_j (K-major)
      const uint32_t idesc_o = make_idesc(1, 1, 0, 1, BQ, D);     // P (K-major) x V_j (MN-major)
      const uint32_t aQ = smem_u32(sQ), aP = smem_u32(sP);
      bool ok = mbar_wait(q_full, 0, abort_flag, p.status, 1200);
      auto issue_s = [&](int it) {
        const int st = it & 1;
        const uint32_t aK = smem_u32(sK + st * kKVBytes);
        const uint32_t d = tmem_S + static_cast<uint32_t>((it & 1) * BKV);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t qoff = (k >> 2) * kQHalf + (k & 3) * 32;
          const uint32_t koff = (k >> 2) * kKVHalf + (k & 3) * 32;
          umma_f16_ss(d, make_smem_desc_sw128(aQ + qoff, 16, 1024), make_smem_desc_sw128(aK + koff, 16, 1024), idesc_s,
                      k != 0 ? 1u : 0u);
        }
        tc_commit(&s_full[it & 1]);
      };
      if (ok) {
        ok = mbar_wait(&k_full[0], 0, abort_flag, p.status, 1201);
        if (ok) {
          tc_fence_after();
          issue_s(0);
        }
      }
      for (int it = 0; it < n_kv && ok; ++it) {
        const int st = it & 1;
        const uint32_t ph = (it >> 1) & 1u;
        if (it + 1 < n_kv) {
          ok = mbar_wait(&k_full[(it + 1) & 1], ((it + 1) >> 1) & 1u, abort_flag, p.status, 1202);
          if (!ok) break;
          tc_fence_after();
          issue_s(it + 1);
        }
        ok = mbar_wait(p_full, it & 1u, abort_flag, p.status, 1203);
        if (!ok) break;
        ok = mbar_wait(&v_full[st], ph, abort_flag, p.status, 1204);
        if (!ok) break;
        tc_fence_after();
        const uint32_t aV = smem_u32(sV + st * kKVBytes);
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k) {
          // A = P: K-major over keys (64-key halves of 128 rows); B = V_j: [key rows x d], d contiguous -> MN-major,
          // its two 64-column groups kKVHalf apart
          const uint64_t adesc = make_smem_desc_sw128(aP + (k >> 2) * kQHalf + (k & 3) * 32, 16, 1024);
          const uint64_t bdesc = make_smem_desc_sw128(aV + k * (16 * 128), kKVHalf, 1024);
          umma_f16_ss(tmem_O, adesc, bdesc, idesc_o, (it | k) != 0 ? 1u : 0u);
        }
        tc_commit(pv_done);
        tc_commit(&kv_empty[st]);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax / correction / epilogue
    const int q = warp & 3;
    const int r = q * 32 + lane;               // row inside the tile == TMEM lane
    const int qg = q0 + r;                     // global query index
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int it = 0; it < n_kv; ++it) {
      ok = mbar_wait(&s_full[it & 1], (it >> 1) & 1u, abort_flag, p.status, 1300);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t tS = tmem_S + lane_addr + static_cast<uint32_t>((it & 1) * BKV);
      const int k0 = (j_lo + it) * BKV;
      const int k_hi = min(qg, p.T - 1);                              // last visible key
      const int k_lo = (p.window < 0) ? 0 : max(0, qg - p.window);    // first visible key
      const bool need_mask = (k0 + BKV - 1 > k_hi) || (k0 < k_lo);
      // The S row is read from TMEM once and stays in registers for both the maximum and the exponentials.
      uint32_t sv[BKV];
#pragma unroll
      for (int ch = 0; ch < BKV / 32; ++ch)
        tmem_ld_32x32(tS + ch * 32, *reinterpret_cast<uint32_t(*)[32]>(sv + ch * 32));
      tc_wait_ld();
      // four independent running maxima (and sums below): one dependent chain of 64 would expose its latency, with only
      // two softmax warps per scheduler there is nothing else to issue meanwhile
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (need_mask) {
#pragma unroll
        for (int j = 0; j < BKV; ++j) {
          const int kg = k0 + j;
          if (!(kg <= k_hi && kg >= k_lo)) sv[j] = __float_as_uint(-INFINITY);
          mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(sv[j]));
        }
      } else {
#pragma unroll
        for (int j = 0; j < BKV; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(sv[j]));
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // Lazy reference maximum: the reference point of the exponentials only moves when the row maximum has grown by
      // more than 2^kLazyLog2 since it was set. In between, probabilities are at most 2^kLazyLog2 (exact in bf16's
      // range), alpha is exactly 1 and O needs no rescaling; l and the log-sum-exp use the same reference, so the
      // result is unchanged.
      constexpr float kLazyLog2 = 8.f;
      const float m_cand = fmaxf(m, mx * p.scale_log2);
      const float m_new = (m == -INFINITY || m_cand - m > kLazyLog2) ? m_cand : m;
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
      const float alpha = (m == -INFINITY) ? 0.f : exp2f(m - m_use);
      // probabilities, packed to bf16 (masked entries are -inf -> 0)
      uint32_t pk[BKV / 2];
      float rs4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < BKV; j += 2) {
        const float e0 = exp2f(fmaf(__uint_as_float(sv[j]), p.scale_log2, -m_use));
        const float e1 = exp2f(fmaf(__uint_as_float(sv[j + 1]), p.scale_log2, -m_use));
        const __nv_bfloat162 pb = __floats2bfloat162_rn(e0, e1);
        const float2 back = __bfloat1622float2(pb);      // the sum uses the rounded values the PV product will see
        rs4[(j >> 1) & 3] += back.x + back.y;
        pk[j / 2] = *reinterpret_cast<const uint32_t*>(&pb);
      }
      const float rs = (rs4[0] + rs4[1]) + (rs4[2] + rs4[3]);
      l = l * alpha + rs;
      m = m_new;
      // O and the P buffer are free once the previous P V product has completed
      if (it > 0) {
        ok = mbar_wait(pv_done, (it - 1) & 1u, abort_flag, p.status, 1301);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (!__all_sync(0xffffffffu, alpha == 1.f)) {
          const uint32_t tO = tmem_O + lane_addr;
#pragma unroll 1
          for (int ch = 0; ch < 4; ++ch) {
            uint32_t v[32];
            tmem_ld_32x32(tO + ch * 32, v);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
            tmem_st_32x32(tO + ch * 32, v);
          }
          tc_wait_st();
        }
      }
      // P row -> shared memory (K-major, 128B swizzle): 16 chunks of 8 keys
#pragma unroll
      for (int c = 0; c < BKV / 8; ++c) {
        const uint32_t off = sw128_offset(r, c * 8, kQHalf);
        *reinterpret_cast<uint4*>(sP + off) = make_uint4(pk[c * 4], pk[c * 4 + 1], pk[c * 4 + 2], pk[c * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(p_full);
    }
    if (ok) {
      ok = mbar_wait(pv_done, (n_kv - 1) & 1u, abort_flag, p.status, 1302);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      const float inv = (l > 0.f) ? 1.f / l : 0.f;
      const uint32_t tO = tmem_O + lane_addr;
      const bool row_ok = qg < p.T;
      __nv_bfloat16* orow = p.out + (((size_t)b * p.T + (row_ok ? qg : 0)) * p.H + h) * D;
#pragma unroll 1
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t v[32];
        tmem_ld_32x32(tO + ch * 32, v);
        tc_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            uint4 t;
            __nv_bfloat162* hh = reinterpret_cast<__nv_bfloat162*>(&t);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              hh[e] = __floats2bfloat162_rn(__uint_as_float(v[j + 2 * e]) * inv, __uint_as_float(v[j + 2 * e + 1]) * inv);
            *reinterpret_cast<uint4*>(orow + ch * 32 + j) = t;
          }
        }
      }
      if (row_ok) p.lse[((size_t)b * p.H + h) * p.T + qg] = (l > 0.f) ? (m * 0.6931471805599453f + logf(l)) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C_::kTmemCols);
  }
}


// ---------------------------------------------------------------------------------------------- two query tiles per CTA
// One CTA per SM and 256 query rows (two 128-row tiles that share every K / V tile of 128 keys). A 128 x 128 tile costs
// 1024 tensor-pipe cycles (QK^T and PV) and 1024 cycles of the special-function pipe, and its softmax cannot start before
// its QK^T has ended nor its PV before the softmax: with two tiles in flight the products of one run under the softmax of
// the other. The issuer's order is  PV0_j S0_{j+1} | PV1_j S1_{j+1}.
//   TMEM   S0 S1 (128 columns each, fp32) and O0 O1 = all 512 columns. P_t (bf16) overlays S_t and is PV's TMEM operand,
//          so the probabilities touch no shared memory and need no proxy fence.
//   shared Q 64 KB + a ring of 5 K / V tiles (32 KB each)
//   warp 0 TMA, warp 1 MMA issuer, warps 4..7 / 8..11 softmax of tile 0 / 1 (one query row per thread: no shuffles);
//   the commit behind S_{j+1} also covers PV_j, so a softmax warp that sees S_{j+1} may touch O.
constexpr int kPairThreads = 384;
constexpr int kPairStages = 5;
constexpr uint32_t kPairTile = 128 * D * 2;
constexpr int kPairSmemBytes = (2 + kPairStages) * kPairTile + 256;

struct TileRange {
  int lo, hi;   // key tiles lo .. hi (inclusive); empty when the tile lies past the end of the sequence
};
__device__ __forceinline__ TileRange pair_range(int q0, int T, int window) {
  if (q0 >= T) return TileRange{1 << 30, -1};
  return TileRange{window < 0 ? 0 : max(0, q0 - window) / 128, min(q0 + 127, T - 1) / 128};
}

// exp2(x * scale - m) of 32 scores, packed to bf16 pairs; adds the rounded values (what PV multiplies) into rs.
__device__ __forceinline__ void exp_chunk(const uint32_t* s, uint64_t sc2, uint64_t nm2, uint32_t (&pk)[16], uint64_t (&rs)[2]) {
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(s[j]), __uint_as_float(s[j + 1])), sc2, nm2);
    float x0, x1;
    unpack_f32x2(x, x0, x1);
    const uint32_t pb = pack_bf16x2(exp2f(x0), exp2f(x1));
    pk[j / 2] = pb;
    rs[(j >> 1) & 1] = add_f32x2(rs[(j >> 1) & 1], pack_f32x2(__uint_as_float(pb << 16), __uint_as_float(pb & 0xffff0000u)));
  }
}

__global__ void __launch_bounds__(kPairThreads, 1)
flash_fwd_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const FwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                          // 2 tiles
  uint8_t* sKV = smem + 2 * kPairTile;         // K_lo V_lo K_lo+1 V_lo+1 ... through the ring
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (2 + kPairStages) * kPairTile);
  uint64_t* q_full = bars;                     // 2
  uint64_t* kv_full = bars + 2;                // kPairStages
  uint64_t* kv_empty = bars + 2 + kPairStages; // kPairStages
  uint64_t* s_full = bars + 2 + 2 * kPairStages;   // 2: S_t ready (and every earlier product of the CTA done)
  uint64_t* p_full = s_full + 2;               // 2 x 2 (count 128): first / second 64 keys of P_t written
  uint64_t* o_full = p_full + 4;               // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_qt = (p.T + 255) / 256;
  const int qt = n_qt - 1 - static_cast<int>(blockIdx.x);   // heavy (late) tiles first
  const int bh = blockIdx.y;
  const int b = bh / p.H, h = bh - b * p.H;
  const int q0 = qt * 256;
  const TileRange r0 = pair_range(q0, p.T, p.window), r1 = pair_range(q0 + 128, p.T, p.window);
  const int j_lo = r0.lo, j_hi = max(r0.hi, r1.hi);          // tile 0 always has rows

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&o_full[i], 1);
      mbar_init(&p_full[2 * i], 128);
      mbar_init(&p_full[2 * i + 1], 128);
    }
    for (int i = 0; i < kPairStages; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    *abort_flag = 0;
    if ((smem_u32(smem) & 1023u) != 0u) report_error(p.status, SR_ERR_BAD_ARG, 1500, 0);   // swizzle needs 1 KB alignment
    fence_barrier_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base, tmem_O = tmem_base + 256;   // + 128 for tile 1

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int st = 0;
      uint32_t ph = 1;
      bool ok = true;
      auto load_kv = [&](const CUtensorMap* map, int j) {
        ok = mbar_wait(&kv_empty[st], ph, abort_flag, p.status, 1600);
        if (!ok) return;
        uint8_t* dst = sKV + st * kPairTile;
        mbar_arrive_expect_tx(&kv_full[st], kPairTile);
        tma_load_4d(dst, map, &kv_full[st], 0, h, j * 128, b);
        tma_load_4d(dst + kQHalf, map, &kv_full[st], 64, h, j * 128, b);
        if (++st == kPairStages) {
          st = 0;
          ph ^= 1u;
        }
      };
      auto load_q = [&](int t) {
        mbar_arrive_expect_tx(&q_full[t], kPairTile);
        tma_load_4d(sQ + t * kPairTile, &map_q, &q_full[t], 0, h, q0 + t * 128, b);
        tma_load_4d(sQ + t * kPairTile + kQHalf, &map_q, &q_full[t], 64, h, q0 + t * 128, b);
      };
      load_q(0);
      load_kv(&map_k, j_lo);
      if (r1.hi >= 0) load_q(1);
      for (int j = j_lo; ok; ) {
        load_kv(&map_v, j);
        if (++j > j_hi || !ok) break;
        load_kv(&map_k, j);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc(1, 1, 0, 0, 128, 128);   // Q (K-major) x K_j (K-major)
      const uint32_t idesc_o = make_idesc(1, 1, 0, 1, 128, D);     // P (TMEM) x V_j (MN-major)
      bool ok = true;
      auto slot = [&](int n) { return sKV + (n % kPairStages) * kPairTile; };   // n-th tile of the ring
      auto wait_slot = [&](int n, int site) {
        ok = mbar_wait(&kv_full[n % kPairStages], (n / kPairStages) & 1u, abort_flag, p.status, site);
        if (ok) tc_fence_after();
        return ok;
      };
      auto issue_s = [&](int t, int n) {
        const uint32_t aQ = smem_u32(sQ + t * kPairTile), aK = smem_u32(slot(n));
        const uint32_t d = tmem_S + t * 128;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k >> 2) * kQHalf + (k & 3) * 32;
          umma_f16_ss(d, make_smem_desc_sw128(aQ + off, 16, 1024), make_smem_desc_sw128(aK + off, 16, 1024), idesc_s, k != 0 ? 1u : 0u);
        }
        tc_commit(&s_full[t]);
      };
      int n = 0;                       // ring position of K_j; V_j is n + 1, K_{j+1} is n + 2
      uint32_t pph0 = 0, pph1 = 0;     // phase of P_0 / P_1
      if (wait_slot(0, 1700)) {
        ok = mbar_wait(&q_full[0], 0, abort_flag, p.status, 1701);
        if (ok) {
          tc_fence_after();
          issue_s(0, 0);
          if (r1.hi >= 0) {
            ok = mbar_wait(&q_full[1], 0, abort_flag, p.status, 1702);
            if (ok && r1.lo == j_lo) {
              tc_fence_after();
              issue_s(1, 0);
            }
          }
          if (ok) tc_commit(&kv_empty[0]);
        }
      }
      for (int j = j_lo; j <= j_hi && ok; ++j, n += 2) {
        if (!wait_slot(n + 1, 1703)) break;
        if (j < j_hi && !wait_slot(n + 2, 1704)) break;
        const uint32_t aV = smem_u32(slot(n + 1));
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const TileRange r = t == 0 ? r0 : r1;
          uint32_t& pph = t == 0 ? pph0 : pph1;
          if (j >= r.lo && j <= r.hi) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              ok = mbar_wait(&p_full[2 * t + half], pph, abort_flag, p.status, 1705 + half);
              if (!ok) break;
              tc_fence_after();
#pragma unroll
              for (int k = half * 4; k < half * 4 + 4; ++k)
                umma_f16_ts(tmem_O + t * 128, tmem_S + t * 128 + k * 8, make_smem_desc_sw128(aV + k * 2048, kQHalf, 1024), idesc_o,
                            (j > r.lo || k != 0) ? 1u : 0u);
            }
            if (!ok) break;
            pph ^= 1u;
            if (j == r.hi) tc_commit(&o_full[t]);
          }
          if (j + 1 >= r.lo && j + 1 <= r.hi) issue_s(t, n + 2);   // overwrites P_t of tile j: products of one issuer run in order
        }
        if (!ok) break;
        tc_commit(&kv_empty[(n + 1) % kPairStages]);
        if (j < j_hi) tc_commit(&kv_empty[(n + 2) % kPairStages]);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ softmax / rescale / epilogue
    const int t = (warp - 4) >> 2;
    const int r = (warp & 3) * 32 + lane;       // row inside the tile == TMEM lane
    const int qb = q0 + t * 128;                // first row of the tile
    const int qg = qb + r;                      // global query index
    const TileRange kr = t == 0 ? r0 : r1;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem_S + t * 128 + lane_addr, tO = tmem_O + t * 128 + lane_addr;
    const int k_hi = min(qg, p.T - 1);                              // last visible key
    const int k_lo = (p.window < 0) ? 0 : max(0, qg - p.window);    // first visible key
    const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    uint32_t ph = 0;
    for (int j = kr.lo; j <= kr.hi; ++j, ph ^= 1u) {
      ok = mbar_wait(&s_full[t], ph, abort_flag, p.status, 1800);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t sv[128];
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) tmem_ld_32x32(tS + ch * 32, *reinterpret_cast<uint32_t(*)[32]>(sv + ch * 32));
      tc_wait_ld();
      const int k0 = j * 128;
      if (k0 + 127 > qb || (p.window >= 0 && k0 < qb + 127 - p.window)) {    // the tile is not inside the band of all its rows
#pragma unroll
        for (int c = 0; c < 128; ++c)
          if (k0 + c > k_hi || k0 + c < k_lo) sv[c] = __float_as_uint(-INFINITY);
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 128; c += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) mx4[e] = fmaxf(fmaxf(mx4[e], __uint_as_float(sv[c + e])), __uint_as_float(sv[c + 4 + e]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // Lazy reference maximum, as in flash_fwd_kernel above: it moves only when the row maximum has grown by more than
      // 2^kLazyLog2, so O is rescaled on almost no tile.
      constexpr float kLazyLog2 = 8.f;
      const float m_cand = fmaxf(m, mx * p.scale_log2);
      const float m_new = (m == -INFINITY || m_cand - m > kLazyLog2) ? m_cand : m;
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
      const float alpha = (m == -INFINITY) ? 1.f : exp2f(m - m_use);     // nothing but zeros to rescale before the first visible key
      m = m_new;
      if (j > kr.lo && !__all_sync(0xffffffffu, alpha == 1.f)) {
        l *= alpha;
#pragma unroll 1
        for (int ch = 0; ch < 8; ++ch) {
          uint32_t v[16];
          tmem_ld_32x16(tO + ch * 16, v);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
          tmem_st_32x16(tO + ch * 16, v);
        }
      }
      const uint64_t nm2 = pack_f32x2(-m_use, -m_use);
      uint64_t rs[2] = {0ull, 0ull};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) {
          uint32_t pk[16];
          exp_chunk(sv + half * 64 + c2 * 32, sc2, nm2, pk, rs);
          tmem_st_32x16(tS + half * 32 + c2 * 16, pk);
        }
        tc_wait_st();
        tc_fence_before();
        mbar_arrive(&p_full[2 * t + half]);
      }
      float a0, a1;
      unpack_f32x2(add_f32x2(rs[0], rs[1]), a0, a1);
      l += a0 + a1;
    }
    if (ok && kr.hi >= 0) {
      ok = mbar_wait(&o_full[t], 0, abort_flag, p.status, 1801);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok && kr.hi >= 0) {
      tc_fence_after();
      const float inv = (l > 0.f) ? 1.f / l : 0.f;
      const bool row_ok = qg < p.T;
      __nv_bfloat16* orow = p.out + (((size_t)b * p.T + (row_ok ? qg : 0)) * p.H + h) * D;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t v[32];
        tmem_ld_32x32(tO + ch * 32, v);
        tc_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int e = 0; e < 32; e += 8)
            *reinterpret_cast<uint4*>(orow + ch * 32 + e) =
                make_uint4(pack_bf16x2(__uint_as_float(v[e]) * inv, __uint_as_float(v[e + 1]) * inv),
                           pack_bf16x2(__uint_as_float(v[e + 2]) * inv, __uint_as_float(v[e + 3]) * inv),
                           pack_bf16x2(__uint_as_float(v[e + 4]) * inv, __uint_as_float(v[e + 5]) * inv),
                           pack_bf16x2(__uint_as_float(v[e + 6]) * inv, __uint_as_float(v[e + 7]) * inv));
        }
      }
      if (row_ok) p.lse[((size_t)b * p.H + h) * p.T + qg] = (l > 0.f) ? (m * 0.6931471805599453f + logf(l)) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

namespace sr_attn {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

extern "C" void* sr_driver_encode_tiled(void);   // process-wide handle, gemm_tcgen05.cu

EncodeTiledFn encode_fn() {
  // a driver-API call: the device's context must be current on this thread (see gemm_common.cuh)
  static thread_local bool bound = false;
  if (!bound) {
    cudaFree(nullptr);
    bound = true;
  }
  return reinterpret_cast<EncodeTiledFn>(sr_driver_encode_tiled());
}

// (B, T, H, 128) bf16 tensor with row stride `ld_t` elements between tokens (the head h slice starts at h*128);
// box = 64 columns x `rows` tokens of one head, 128B swizzle, zero fill past T.
int encode_bthd(CUtensorMap* map, const void* ptr, int B, int T, int H, long ld_t, int rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || (ld_t % 8) != 0) return -2;
  cuuint64_t dims[4] = {128, (cuuint64_t)H, (cuuint64_t)T, (cuuint64_t)B};
  cuuint64_t strides[3] = {128 * 2, (cuuint64_t)ld_t * 2, (cuuint64_t)ld_t * 2 * (cuuint64_t)T};
  cuuint32_t box[4] = {64, 1, (cuuint32_t)rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Contiguous (B, T, H, 128) fp32 tensor; box = 32 columns (128 B) x `rows` tokens of one head, 128B swizzle. Used for the
// bulk reduce-add of dQ tiles from shared memory.
int encode_bthd_f32(CUtensorMap* map, const void* ptr, int B, int T, int H, int rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0) return -2;
  cuuint64_t dims[4] = {128, (cuuint64_t)H, (cuuint64_t)T, (cuuint64_t)B};
  cuuint64_t strides[3] = {128 * 4, (cuuint64_t)H * 128 * 4, (cuuint64_t)H * 128 * 4 * (cuuint64_t)T};
  cuuint32_t box[4] = {32, 1, (cuuint32_t)rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

}  // namespace sr_attn

// q, k, v: (B, T, H, 128) bf16 with token stride ld_* elements (contiguous tensors: H*128); out contiguous;
// lse: fp32 (B, H, T), natural log of sum exp(scale * s). window < 0 = full causal.
template <int BKV>
int launch_fwd(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const FwdParams& p, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(flash_fwd_kernel<BKV>, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdCfg<BKV>::kSmemBytes) !=
        cudaSuccess)
      return -4;
    configured = true;
  }
  dim3 grid((p.T + BQ - 1) / BQ, p.B * p.H);
  flash_fwd_kernel<BKV><<<grid, kThreads, FwdCfg<BKV>::kSmemBytes, stream>>>(mq, mk, mv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// q, k, v: (B, T, H, 128) bf16 with token stride ld_* elements (contiguous tensors: H*128); out contiguous;
// lse: fp32 (B, H, T), natural log of sum exp(scale * s). window < 0 = full causal. bkv: 64 or 128 keys per tile.
extern "C" int sr_flash_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int T, int H,
                                 long ld_q, long ld_k, long ld_v, int window, float scale, int bkv, int* status,
                                 cudaStream_t stream) {
  if (B <= 0 || T <= 0 || H <= 0) return 0;
  if (bkv != 64 && bkv != 128) return -2;
  CUtensorMap mq, mk, mv;
  int rc;
  if ((rc = sr_attn::encode_bthd(&mq, q, B, T, H, ld_q, BQ))) return rc;
  if ((rc = sr_attn::encode_bthd(&mk, k, B, T, H, ld_k, bkv))) return rc - 10;
  if ((rc = sr_attn::encode_bthd(&mv, v, B, T, H, ld_v, bkv))) return rc - 20;
  FwdParams p;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.B = B; p.T = T; p.H = H;
  p.window = (window < 0 || window >= T) ? -1 : window;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  if (bkv == 64) return launch_fwd<64>(mq, mk, mv, p, stream);
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(flash_fwd_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemBytes) != cudaSuccess)
      return -4;
    configured = true;
  }
  dim3 grid((p.T + 255) / 256, p.B * p.H);
  flash_fwd_pair_kernel<<<grid, kPairThreads, kPairSmemBytes, stream>>>(mq, mk, mv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
