// Flash attention backward for sm_100a (same problem as flash_attn_fwd.cu): dQ, dK, dV from dO, Q, K, V, O, LSE.
//
// One CTA per (batch*head, 128-key tile j): K_j and V_j stay in shared memory, the CTA walks the query tiles i that can
// see them. Per query tile, five tcgen05 products with fp32 accumulators in TMEM, the score tiles held transposed
// (TMEM lane = key) so that the probabilities never leave TMEM:
//     S^T  = K_j Q_i^T          dP^T = V_j dO_i^T               (both operands K-major)
//     dV  += P^T dO_i           (A = P^T, bf16 in the TMEM columns of S^T; B MN-major)
//     dK  += dS^T Q_i           dQ_i = dS K_j                   (one shared-memory tile dS^T, read K-major and MN-major)
// with P = exp(scale*S - lse) and dS = P * (dP - delta) * scale.
//
// What bounds it: a tile pair is 5 x 512 tensor-pipe cycles, 128*128 exponentials (1024 cycles of the special-function
// pipe) and about 4000 cycles' worth of shared-memory traffic (operands, dS, dQ staging, loads), so the point of the
// layout is to have all three under way at once. The issuer runs
//     dV_i | S_{i+1} | dQ_i | dK_i | dP_{i+1}
// so that the exponentials of tile i+1 (warps 4..11, after S_{i+1}) overlap dQ_i and dK_i, forming dS_i overlaps dV_i and
// S_{i+1}, and dQ_i is drained by warps of its own (12..15) while dK_i runs. P^T shares columns with S^T and dQ with dP^T
// (S/P 128 + dP/dQ 128 + dV 128 + dK 128 = all 512).
//   warp 0       TMA: K, V once; Q through a 2-stage ring (dK_i still reads Q_i when S_{i+1} starts), dO single-buffered
//   warp 1       MMA issuer + TMEM owner
//   warp 2       -lse*log2(e) and -delta of the query rows into shared memory (they vary along the columns of a lane)
//   warps 4..11  P and dS; a lane's 128 columns are split between two threads; afterwards dK / dV epilogue
//   warps 12..15 dQ tile: TMEM -> registers -> 4 KB staging boxes -> bulk tensor reduce-add into the fp32 accumulator
// Measured (CUDA events, L2 flushed, without the fill of the dQ accumulator; before: one role sequence S, dP -> P, dS ->
// dV, dK, dQ -> dQ drain per tile with nothing overlapped): (4, 2048, 20, 128) window 1024 342 -> 225 us (716 TFLOP/s of
// visible work), full causal 428 -> 270 us; (32, 2048, 8, 128) window 1024 1007 -> 664 us; (3, 1000, 5, 128) 35 -> 27 us.
#include "sm100_common.cuh"

namespace sr_attn {
int encode_bthd(CUtensorMap* map, const void* ptr, int B, int T, int H, long ld_t, int rows);
int encode_bthd_f32(CUtensorMap* map, const void* ptr, int B, int T, int H, int rows);
}

namespace {

using namespace sr;

constexpr int BQ = 128, BKV = 128, D = 128;
constexpr int kThreads = 512;
constexpr int kComputeThreads = 256;
constexpr uint32_t kTileBytes = 128 * 128 * 2;
constexpr uint32_t kHalfBytes = 128 * 128;
constexpr uint32_t kStageBytes = 32 * 32 * 4;            // one dQ staging box: 32 rows x 32 fp32 columns
constexpr int kSmemStage = 6 * kTileBytes;               // K, V, Q x 2, dO, dS; then 4 warps x 2 staging boxes
constexpr int kSmemStat = kSmemStage + 8 * kStageBytes;  // 2 stages x (128 x -lse*log2e, 128 x -delta)
constexpr int kSmemBars = kSmemStat + 2 * 2 * 128 * 4;
constexpr int kSmemBytes = kSmemBars + 256;

struct BwdParams {
  const float* lse;      // [B, H, T]
  const float* delta;    // [B, H, T]
  float* dq_acc;         // [B, T, H, D] fp32
  __nv_bfloat16* dk;     // [B, T, H, D]
  __nv_bfloat16* dv;
  int B, T, H, window;
  float scale, scale_log2;
  int* status;
};

// delta[b, h, t] = sum_d dO[b, t, h, d] * O[b, t, h, d]; one warp per (b, t, h)
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O,
                                  float* __restrict__ delta, int B, int T, int H) {
  const long wid = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (wid >= (long)B * T * H) return;
  const int lane = threadIdx.x & 31;
  const uint2 a = *reinterpret_cast<const uint2*>(dO + wid * D + lane * 4);
  const uint2 o = *reinterpret_cast<const uint2*>(O + wid * D + lane * 4);
  const float2 a0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.x));
  const float2 a1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.y));
  const float2 o0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.x));
  const float2 o1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.y));
  float s = a0.x * o0.x + a0.y * o0.y + a1.x * o1.x + a1.y * o1.y;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (lane == 0) {
    const long bt = wid / H;
    const int h = (int)(wid - bt * H);
    const long b = bt / T;
    const int t = (int)(bt - b * T);
    delta[(b * H + h) * T + t] = s;
  }
}

__global__ void attn_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, long n4) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long)gridDim.x * blockDim.x) {
    const float4 v = reinterpret_cast<const float4*>(acc)[i];
    uint2 o;
    *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(v.x, v.y);
    *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(v.z, v.w);
    reinterpret_cast<uint2*>(dq)[i] = o;
  }
}

// smem tile (128B-swizzled box of the fp32 map) += into global memory, tracked by the thread's bulk async-group
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, const void* smem_src, int c0, int c1, int c2,
                                                  int c3) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      ::"l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// P = exp2(S * scale_log2 - lse2) of 32 columns, in place. c_lo / c_hi: visible columns of this lane (MASK only).
template <bool MASK>
__device__ __forceinline__ void probabilities(uint32_t (&s)[32], const float* nlse, float scale_log2, int c_lo, int c_hi) {
  const uint64_t sc2 = pack_f32x2(scale_log2, scale_log2);
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    const ulonglong2 nl = *reinterpret_cast<const ulonglong2*>(nlse + c);
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(s[c + e]), __uint_as_float(s[c + e + 1])), sc2, e == 0 ? nl.x : nl.y);
      float x0, x1;
      unpack_f32x2(x, x0, x1);
      float p0 = exp2f(x0), p1 = exp2f(x1);
      if (MASK) {
        if (c + e < c_lo || c + e > c_hi) p0 = 0.f;
        if (c + e + 1 < c_lo || c + e + 1 > c_hi) p1 = 0.f;
      }
      s[c + e] = __float_as_uint(p0);
      s[c + e + 1] = __float_as_uint(p1);
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                 const __grid_constant__ CUtensorMap map_dq, const BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = smem + kTileBytes;
  uint8_t* sQ = smem + 2 * kTileBytes;    // 2 stages
  uint8_t* sdO = smem + 4 * kTileBytes;
  uint8_t* sdS = smem + 5 * kTileBytes;   // dS^T: row = key, query contiguous
  float* sStat = reinterpret_cast<float*>(smem + kSmemStat);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSmemBars);
  uint64_t* kv_full = bars;          // 1
  uint64_t* q_full = bars + 1;       // 2
  uint64_t* q_empty = bars + 3;      // 2  commit after dK_i
  uint64_t* do_full = bars + 5;      // 1
  uint64_t* do_empty = bars + 6;     // 1  commit after dV_i
  uint64_t* stat_full = bars + 7;    // 2  32 arrivals
  uint64_t* stat_empty = bars + 9;   // 2  256 arrivals
  uint64_t* s_full = bars + 11;      // 1  S^T ready
  uint64_t* dp_full = bars + 12;     // 1  dP^T ready
  uint64_t* p_full = bars + 13;      // 256 arrivals: P^T in TMEM, S^T consumed
  uint64_t* ds_full = bars + 14;     // 256 arrivals: dS^T in shared memory, dP^T consumed
  uint64_t* ds_empty = bars + 15;    // commit after dK_i (and dQ_i): the dS tile may be overwritten
  uint64_t* dq_full = bars + 16;     // commit after dQ_i
  uint64_t* dq_read = bars + 17;     // 128 arrivals: dQ_i is in registers, the dP columns are free
  uint64_t* acc_full = bars + 18;    // commit after the last product
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x;
  const int bh = blockIdx.y;
  const int b = bh / p.H, h = bh - b * p.H;
  const int k0 = j * BKV;
  const int n_qt = (p.T + BQ - 1) / BQ;
  const int i_lo = j;   // BQ == BKV: the diagonal tile
  int i_hi = n_qt - 1;
  if (p.window >= 0) i_hi = min(i_hi, (min(k0 + BKV - 1, p.T - 1) + p.window) / BQ);
  const int n_q = i_hi - i_lo + 1;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&stat_full[i], 32);
      mbar_init(&stat_empty[i], kComputeThreads);
    }
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, kComputeThreads);
    mbar_init(ds_full, kComputeThreads);
    mbar_init(ds_empty, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_read, 128);
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    if ((smem_u32(smem) & 1023u) != 0u) report_error(p.status, SR_ERR_BAD_ARG, 2000, 0);   // swizzle needs 1 KB alignment
    fence_barrier_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_do);
    tma_prefetch_desc(&map_dq);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 384;
  const uint32_t tdQ = tdP;  // the dP columns are reused for the dQ tile once dP has been consumed
  // P^T (bf16 pairs) overlays S^T: queries 0..63 in columns 0..31, queries 64..127 in columns 64..95, so that each of the
  // two threads of a lane only overwrites scores that it has read itself.

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_arrive_expect_tx(kv_full, 2 * kTileBytes);
      tma_load_4d(sK, &map_k, kv_full, 0, h, k0, b);
      tma_load_4d(sK + kHalfBytes, &map_k, kv_full, 64, h, k0, b);
      tma_load_4d(sV, &map_v, kv_full, 0, h, k0, b);
      tma_load_4d(sV + kHalfBytes, &map_v, kv_full, 64, h, k0, b);
      for (int it = 0; it < n_q; ++it) {
        const int st = it & 1;
        const int q0 = (i_lo + it) * BQ;
        if (!mbar_wait(&q_empty[st], ((it >> 1) & 1u) ^ 1u, abort_flag, p.status, 2100)) break;
        uint8_t* dst = sQ + st * kTileBytes;
        mbar_arrive_expect_tx(&q_full[st], kTileBytes);
        tma_load_4d(dst, &map_q, &q_full[st], 0, h, q0, b);
        tma_load_4d(dst + kHalfBytes, &map_q, &q_full[st], 64, h, q0, b);
        if (!mbar_wait(do_empty, (it & 1u) ^ 1u, abort_flag, p.status, 2101)) break;
        mbar_arrive_expect_tx(do_full, kTileBytes);
        tma_load_4d(sdO, &map_do, do_full, 0, h, q0, b);
        tma_load_4d(sdO + kHalfBytes, &map_do, do_full, 64, h, q0, b);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t id_kk = make_idesc(1, 1, 0, 0, 128, 128);   // K-major x K-major
      const uint32_t id_mm = make_idesc(1, 1, 1, 1, 128, 128);   // MN-major x MN-major
      const uint32_t id_km = make_idesc(1, 1, 0, 1, 128, 128);   // K-major (or TMEM) x MN-major
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), adO = smem_u32(sdO), adS = smem_u32(sdS);
      auto kmaj = [&](uint32_t base, int k) { return make_smem_desc_sw128(base + (k >> 2) * kHalfBytes + (k & 3) * 32, 16, 1024); };
      auto mnmaj = [&](uint32_t base, int k) { return make_smem_desc_sw128(base + k * 2048, kHalfBytes, 1024); };
      auto issue_s = [&](int it) {
        const uint32_t aQ = smem_u32(sQ + (it & 1) * kTileBytes);
#pragma unroll
        for (int k = 0; k < 8; ++k) umma_f16_ss(tS, kmaj(aK, k), kmaj(aQ, k), id_kk, k != 0 ? 1u : 0u);
        tc_commit(s_full);
      };
      auto issue_dp = [&]() {
#pragma unroll
        for (int k = 0; k < 8; ++k) umma_f16_ss(tdP, kmaj(aV, k), kmaj(adO, k), id_kk, k != 0 ? 1u : 0u);
        tc_commit(dp_full);
      };
      bool ok = mbar_wait(kv_full, 0, abort_flag, p.status, 2200) && mbar_wait(&q_full[0], 0, abort_flag, p.status, 2201);
      if (ok) {
        tc_fence_after();
        issue_s(0);
        ok = mbar_wait(do_full, 0, abort_flag, p.status, 2202);
      }
      if (ok) {
        tc_fence_after();
        issue_dp();
      }
      for (int it = 0; it < n_q && ok; ++it) {
        const uint32_t ph = it & 1u;
        const bool more = it + 1 < n_q;
        ok = mbar_wait(p_full, ph, abort_flag, p.status, 2203);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_f16_ts(tdV, tS + (k >> 2) * 64 + (k & 3) * 8, mnmaj(adO, k), id_km, (it | k) != 0 ? 1u : 0u);
        tc_commit(do_empty);
        if (more) {   // overwrites P_i: products of one issuer execute in order
          ok = mbar_wait(&q_full[(it + 1) & 1], ((it + 1) >> 1) & 1u, abort_flag, p.status, 2204);
          if (!ok) break;
          tc_fence_after();
          issue_s(it + 1);
        }
        ok = mbar_wait(ds_full, ph, abort_flag, p.status, 2205);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k) umma_f16_ss(tdQ, mnmaj(adS, k), mnmaj(aK, k), id_mm, k != 0 ? 1u : 0u);
        tc_commit(dq_full);
        const uint32_t aQ = smem_u32(sQ + (it & 1) * kTileBytes);
#pragma unroll
        for (int k = 0; k < 8; ++k) umma_f16_ss(tdK, kmaj(adS, k), mnmaj(aQ, k), id_km, (it | k) != 0 ? 1u : 0u);
        tc_commit(&q_empty[it & 1]);
        tc_commit(ds_empty);
        if (more) {
          ok = mbar_wait(do_full, ph ^ 1u, abort_flag, p.status, 2206) && mbar_wait(dq_read, ph, abort_flag, p.status, 2207);
          if (!ok) break;
          tc_fence_after();
          issue_dp();
        }
      }
      if (ok) tc_commit(acc_full);
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ row statistics
    const float log2e = 1.4426950408889634f;
    const size_t base = ((size_t)b * p.H + h) * p.T;
    for (int it = 0; it < n_q; ++it) {
      const int st = it & 1;
      const int q0 = (i_lo + it) * BQ;
      float l[4], d[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int qg = q0 + e * 32 + lane;
        const bool row_ok = qg < p.T;
        l[e] = row_ok ? -p.lse[base + qg] * log2e : -INFINITY;   // rows past the end: every probability is exp2(-inf) = 0
        d[e] = row_ok ? -p.delta[base + qg] : 0.f;
      }
      bool ok = mbar_wait(&stat_empty[st], ((it >> 1) & 1u) ^ 1u, abort_flag, p.status, 2400);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      float* dst = sStat + st * 256;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        dst[e * 32 + lane] = l[e];
        dst[128 + e * 32 + lane] = d[e];
      }
      mbar_arrive(&stat_full[st]);
    }
  } else if (warp >= 4 && warp < 12) {
    // ------------------------------------------------------------------ P and dS
    const int q = warp & 3;                 // TMEM lane quarter this warp may access
    const int chalf = (warp - 4) >> 2;      // which 64 query columns of the lane this thread handles
    const int r = q * 32 + lane;            // key row inside the tile == TMEM lane
    const int kg = k0 + r;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t tS_half = tS + lane_addr + chalf * 64, tdP_half = tdP + lane_addr + chalf * 64;
    bool ok = true;
    for (int it = 0; it < n_q; ++it) {
      const uint32_t ph = it & 1u;
      const int st = it & 1;
      const int q0 = (i_lo + it) * BQ;
      ok = mbar_wait(&stat_full[st], (it >> 1) & 1u, abort_flag, p.status, 2300) &&
           mbar_wait(s_full, ph, abort_flag, p.status, 2301);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      // tiles strictly inside the visible band need no per-element mask (most tiles of a long sequence)
      const bool tile_full = (k0 + BKV - 1 <= q0) && (p.window < 0 || q0 + BQ - 1 <= k0 + p.window);
      const int c_lo = kg - (q0 + chalf * 64);                               // first and last query column that sees this key
      const int c_hi = (p.window < 0) ? 1 << 20 : c_lo + p.window;
      const float* nlse = sStat + st * 256 + chalf * 64;
      uint32_t s0[32], s1[32];
      tmem_ld_32x32(tS_half, s0);
      tmem_ld_32x32(tS_half + 32, s1);
      tc_wait_ld();
      if (tile_full) {
        probabilities<false>(s0, nlse, p.scale_log2, 0, 0);
        probabilities<false>(s1, nlse + 32, p.scale_log2, 0, 0);
      } else {
        probabilities<true>(s0, nlse, p.scale_log2, c_lo, c_hi);
        probabilities<true>(s1, nlse + 32, p.scale_log2, c_lo - 32, c_hi - 32);
      }
      {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = pack_bf16x2(__uint_as_float(s0[2 * e]), __uint_as_float(s0[2 * e + 1]));
        tmem_st_32x16(tS_half, pk);
#pragma unroll
        for (int e = 0; e < 16; ++e) pk[e] = pack_bf16x2(__uint_as_float(s1[2 * e]), __uint_as_float(s1[2 * e + 1]));
        tmem_st_32x16(tS_half + 16, pk);
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(p_full);
      ok = mbar_wait(dp_full, ph, abort_flag, p.status, 2302) &&
           (it == 0 || mbar_wait(ds_empty, ph ^ 1u, abort_flag, p.status, 2303));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float* ndelta = nlse + 128;
      const uint64_t sc2 = pack_f32x2(p.scale, p.scale);
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t dp[16];
        tmem_ld_32x16(tdP_half + ch * 16, dp);
        tc_wait_ld();
        uint32_t dd[8];
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
          const ulonglong2 nd = *reinterpret_cast<const ulonglong2*>(ndelta + ch * 16 + c);
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const int cc = (ch & 1) * 16 + c + e;
            const uint32_t pa = ch < 2 ? s0[cc] : s1[cc], pb = ch < 2 ? s0[cc + 1] : s1[cc + 1];
            const uint64_t t = add_f32x2(pack_f32x2(__uint_as_float(dp[c + e]), __uint_as_float(dp[c + e + 1])), e == 0 ? nd.x : nd.y);
            float d0, d1;
            unpack_f32x2(mul_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(pa), __uint_as_float(pb)), t), sc2), d0, d1);
            dd[(c + e) / 2] = pack_bf16x2(d0, d1);
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
          *reinterpret_cast<uint4*>(sdS + sw128_offset(r, chalf * 64 + ch * 16 + c * 8, kHalfBytes)) =
              make_uint4(dd[c * 4], dd[c * 4 + 1], dd[c * 4 + 2], dd[c * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(ds_full);
      mbar_arrive(&stat_empty[st]);
    }
    // ---- dK / dV epilogue
    if (ok) {
      ok = mbar_wait(acc_full, 0, abort_flag, p.status, 2304);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      const bool row_ok = kg < p.T;
      const size_t base = (((size_t)b * p.T + (row_ok ? kg : 0)) * p.H + h) * D;
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint32_t t = (which == 0 ? tdV : tdK) + lane_addr;
        __nv_bfloat16* dstp = (which == 0 ? p.dv : p.dk) + base;
#pragma unroll 1
        for (int ch = chalf * 2; ch < chalf * 2 + 2; ++ch) {
          uint32_t v[32];
          tmem_ld_32x32(t + ch * 32, v);
          tc_wait_ld();
          if (row_ok) {
#pragma unroll
            for (int jj = 0; jj < 32; jj += 8) {
              uint4 o;
              uint32_t* hh = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
              for (int e = 0; e < 4; ++e)
                hh[e] = pack_bf16x2(__uint_as_float(v[jj + 2 * e]), __uint_as_float(v[jj + 2 * e + 1]));
              *reinterpret_cast<uint4*>(dstp + ch * 32 + jj) = o;
            }
          }
        }
      }
    }
  } else if (warp >= 12) {
    // ------------------------------------------------------------------ dQ tile -> fp32 accumulator in global memory
    const int q = warp & 3;
    const uint32_t tq = tdQ + (static_cast<uint32_t>(q * 32) << 16);
    uint8_t* stage = smem + kSmemStage + (warp - 12) * 2 * kStageBytes;
    for (int it = 0; it < n_q; ++it) {
      const int row0 = (i_lo + it) * BQ + q * 32;
      bool ok = mbar_wait(dq_full, it & 1u, abort_flag, p.status, 2500);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[2][32];
        tmem_ld_32x32(tq + half * 64, v[0]);
        tmem_ld_32x32(tq + half * 64 + 32, v[1]);
        tc_wait_ld();
        if (half == 1) {
          tc_fence_before();
          mbar_arrive(dq_read);
        }
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) {
          uint8_t* box = stage + c2 * kStageBytes;
          if (lane == 0) bulk_wait_read<1>();     // the reduce-add issued from this box two steps ago has read it
          __syncwarp();
          uint8_t* rowp = box + lane * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(rowp + ((c ^ (lane & 7)) << 4)) =
                make_uint4(v[c2][4 * c], v[c2][4 * c + 1], v[c2][4 * c + 2], v[c2][4 * c + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (row0 < p.T) tma_reduce_add_4d(&map_dq, box, half * 64 + c2 * 32, h, row0, b);   // rows past T are clipped
            bulk_commit_group();
          }
        }
      }
    }
    if (lane == 0) bulk_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

// All tensors contiguous (B, T, H, 128) bf16 except lse/delta fp32 (B, H, T) and dq_acc fp32 (B, T, H, 128), which must
// be zero on entry. window < 0 = full causal.
// flags: bit 0 = `delta` already holds rowsum(dO * O) (skip the pre-pass); bit 1 = leave dQ in `dq_acc` (fp32), do not
// write `dq`.
extern "C" int sr_flash_attn_bwd_ex(const void* dO, const void* q, const void* k, const void* v, const void* out,
                                    const float* lse, float* delta, float* dq_acc, void* dq, void* dk, void* dv, int B,
                                    int T, int H, int window, float scale, int flags, int* status, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || H <= 0) return 0;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(flash_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess)
      return -4;
    configured = true;
  }
  const long ld = (long)H * D;
  CUtensorMap mq, mk, mv, mdo;
  int rc;
  if ((rc = sr_attn::encode_bthd(&mq, q, B, T, H, ld, 128))) return rc;
  if ((rc = sr_attn::encode_bthd(&mk, k, B, T, H, ld, 128))) return rc - 10;
  if ((rc = sr_attn::encode_bthd(&mv, v, B, T, H, ld, 128))) return rc - 20;
  if ((rc = sr_attn::encode_bthd(&mdo, dO, B, T, H, ld, 128))) return rc - 30;
  CUtensorMap mdq;
  if ((rc = sr_attn::encode_bthd_f32(&mdq, dq_acc, B, T, H, 32))) return rc - 40;
  const long rows = (long)B * T * H;
  if (!(flags & 1))
    attn_delta_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(dO),
                                                                       reinterpret_cast<const __nv_bfloat16*>(out), delta, B, T, H);
  BwdParams p;
  p.lse = lse; p.delta = delta; p.dq_acc = dq_acc;
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk);
  p.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  p.B = B; p.T = T; p.H = H;
  p.window = (window < 0 || window >= T) ? -1 : window;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  dim3 grid((T + BKV - 1) / BKV, B * H);
  flash_bwd_kernel<<<grid, kThreads, kSmemBytes, stream>>>(mq, mk, mv, mdo, mdq, p);
  if (!(flags & 2)) {
    const long n4 = rows * D / 4;
    long blocks = (n4 + 255) / 256;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (blocks > (long)sms * 16) blocks = (long)sms * 16;
    attn_dq_convert_kernel<<<(unsigned)blocks, 256, 0, stream>>>(dq_acc, reinterpret_cast<__nv_bfloat16*>(dq), n4);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int sr_flash_attn_bwd(const void* dO, const void* q, const void* k, const void* v, const void* out,
                                 const float* lse, float* delta, float* dq_acc, void* dq, void* dk, void* dv, int B, int T,
                                 int H, int window, float scale, int* status, cudaStream_t stream) {
  return sr_flash_attn_bwd_ex(dO, q, k, v, out, lse, delta, dq_acc, dq, dk, dv, B, T, H, window, scale, 0, status, stream);
}
