// Fused causal self-attention (flash-attention style) on tcgen05 tensor cores.
//
// Replaces the reference's attention chain -- QKV split, four transposes, a batched
// matmul that materialises the [B,H,T,T] scores, scale, mask, softmax, a second
// batched matmul and a transpose back (example/gpt2/net.cc:77-108; kernels
// split.cu, transform.cu, softmax.cu, linear.cu) -- with one forward and one
// backward kernel that keep the score tile in tensor memory:
//
//   forward, one CTA per (128 query rows, head, batch), loop over key blocks j <= i:
//     S = Q K_j^T          tcgen05.mma, A/B from TMA-loaded swizzled smem, D in TMEM
//     online softmax       128 threads, one score row each, read with tcgen05.ld
//     P -> smem (bf16)     written in the 128-byte-swizzle layout the MMA expects
//     O_blk = P V_j        tcgen05.mma with V as an MN-major operand (no transpose)
//     O = O * alpha + O_blk in registers; finally O / l and the log-sum-exp row.
//
//   backward, one CTA per (128 key rows, kv head, batch), loop over query blocks i >= j
//   and over the query heads that share the kv head (GQA):
//     S^T = K_j Q_i^T, dP^T = V_j dO_i^T        -> TMEM
//     P = exp(S - lse), dS = P (dP - delta)     -> P^T (bf16) in TMEM, dS^T (bf16) in smem, read as
//                                                  a K-major and as an MN-major operand
//     dV += P^T dO_i, dK += dS^T Q_i            accumulate in TMEM over the whole loop
//     dQ_i += dS K_j                            TMEM -> smem -> fp32 TMA reduce-adds in HBM
//
// q/k/v are addressed in place inside a fused projection buffer through TMA tensor
// maps (row stride = token stride), so no split/transpose kernel runs.  All waits
// are bounded (ptx_sm100.cuh).
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>

#include "api.h"
#include "ptx_sm100.cuh"

namespace titb {

bool make_tmap_tokens(CUtensorMap* m, const void* base, int fp32, uint64_t width, uint64_t T, uint64_t B, uint64_t ld,
                      uint32_t box_width, uint32_t box_tokens);

constexpr int kAttnThreads = 192;
constexpr int kBlk = 128;             // query rows per CTA tile and keys per step
constexpr int kChunkBytes = kBlk * 128;  // one [128 rows x 64 bf16] swizzled sub-tile
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Byte offset of 8 consecutive bf16 (one 16-byte unit) in a [128 x 128] tile stored as two
// [128 rows x 128 B] sub-tiles with the 128-byte swizzle: unit index u = col / 8 in 0..15.
__device__ __forceinline__ uint32_t swz_off(int row, int u) {
  return static_cast<uint32_t>((u >> 3) * kChunkBytes + row * 128 + (((u & 7) ^ (row & 7)) << 4));
}

// A shared-memory descriptor whose start address is moved by `bytes` (a multiple of 16 that stays inside the CTA's
// shared memory): only the 14-bit address field changes, so one add replaces rebuilding the descriptor.
__device__ __forceinline__ uint64_t desc_add(uint64_t desc, uint32_t bytes) { return desc + (bytes >> 4); }

struct AttnArgs {
  int B, T, Hq, Hkv, hd;
  float scale;
  bf16* o;
  float* lse;
  long long o_stride_t;
  // backward
  const float* delta;
  float* dq_accum;  // fp32 [B, T, Hq, hd]
  bf16* dk;
  bf16* dv;
  long long dk_stride_t, dv_stride_t;
  int* status;
};

// ------------------------------------------------------------------------- forward
template <int HD>
struct FwdCfg {
  static constexpr int kTileBytes = kBlk * HD * 2;  // Q, K or V tile
  static constexpr int kStages = 2;
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + kTileBytes;
  static constexpr int kV = kK + kStages * kTileBytes;
  static constexpr int kP = kV + kStages * kTileBytes;
  static constexpr int kBar = kP + kBlk * kBlk * 2;
  static constexpr int kSmem = kBar + 128;
  static constexpr int kTmemCols = 256;  // S: [0,128)  O_blk: [128, 128+HD)
};

// Forward pipeline.  Per key block j the CTA runs
//   MMA warp:      S(j+1) = Q K(j+1)^T is issued as soon as the softmax warps have copied S(j) out of tensor
//                  memory (s_free), i.e. it runs underneath the exponentials of block j; O += P(j) V(j) is issued
//                  when P(j) has been written (p_full) and accumulates in tensor memory over the whole loop.
//   softmax warps: one score row per thread, read from tensor memory ONCE (128 registers), row maximum, then the
//                  exponentials straight from registers.  The running maximum `m_ref` that the exponentials refer
//                  to is only advanced when a block's maximum exceeds it by more than 2^8 (P stays within bf16
//                  range, the row sum is fp32); only then is the O accumulator rescaled, in place in tensor
//                  memory, after the previous P V product has finished.  P(j) is stored to shared memory after
//                  P(j-1) V(j-1) has finished reading the buffer.
// The exponents, their sum and the maximum take half an instruction per score (packed fp32 pairs, three-way maximum); the
// longest rows of tiles of all heads start first, so that the last wave is made of short ones.  Bound: 1024 cycles of
// exponentials per block and SM, with the chain S -> maximum -> exponentials -> P of two CTAs (hd 64) to hide it.
// Measured (B200; before = scalar, tiles of one head in a row): 8 x 1024, 12 heads, hd 64: 39.6 -> 32.3 us; 1 x 1999, 32 / 8
// heads: 48.8 -> 33.4 us; 4 x 2048: 138 -> 117 us; hd 128, 1 x 4096, 32 / 8 heads: 174 -> 153 us (897 TFLOP/s).
template <int HD>
__global__ void __launch_bounds__(kAttnThreads, (HD == 64) ? 2 : 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                const __grid_constant__ CUtensorMap tv, const AttnArgs p) {
  using Cfg = FwdCfg<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kBar);
  uint64_t* q_full = bars;          // 1
  uint64_t* k_full = bars + 1;      // [2]
  uint64_t* k_empty = bars + 3;     // [2]  a K tile is free as soon as its S product has finished ...
  uint64_t* v_full = bars + 5;      // [2]
  uint64_t* v_empty = bars + 7;     // [2]  ... a V tile only after its P V product: K runs a block further ahead
  uint64_t* s_full = bars + 9;
  uint64_t* p_full = bars + 10;
  uint64_t* o_full = bars + 11;
  uint64_t* s_free = bars + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  const int nqb = (p.T + kBlk - 1) / kBlk;
  const int qb = nqb - 1 - blockIdx.y;  // the longest rows of tiles of all heads start first
  const int h = blockIdx.x % p.Hq, b = blockIdx.x / p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  const int q0 = qb * kBlk;
  const int nblk = qb + 1;

  if (threadIdx.x == 0) {
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&k_full[s], 1); ptx::mbar_init(&k_empty[s], 1);
      ptx::mbar_init(&v_full[s], 1); ptx::mbar_init(&v_empty[s], 1);
    }
    ptx::mbar_init(s_full, 1);
    ptx::mbar_init(p_full, 4);
    ptx::mbar_init(o_full, 1);
    ptx::mbar_init(s_free, 4);
    *abort_flag = (ptx::smem_u32(smem) & 1023u) ? 1u : 0u;  // swizzled tiles need a 1024-byte aligned base
    ptx::mbar_fence_init();
    ptx::tma_prefetch_desc(&tq);
    ptx::tma_prefetch_desc(&tk);
    ptx::tma_prefetch_desc(&tv);
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, Cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependency_wait();
  dependents_launch();
  const uint32_t tS = tmem_base, tO = tmem_base + 128;
  const bool bad_align = (*abort_flag != 0);

  if (bad_align) {
    // fall through to the common exit
  } else if (warp == 0) {
    if (ptx::elect_one()) {
      ptx::mbar_expect_tx(q_full, Cfg::kTileBytes);
#pragma unroll
      for (int c = 0; c < HD / 64; ++c)
        ptx::tma_load_3d(smem + Cfg::kQ + c * kChunkBytes, &tq, q_full, h * HD + c * 64, q0, b);
      for (int j = 0; j < nblk; ++j) {
        const int st = j & 1;
        if (!ptx::mbar_wait(&k_empty[st], ((j >> 1) & 1) ^ 1u, abort_flag)) break;
        ptx::mbar_expect_tx(&k_full[st], Cfg::kTileBytes);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          ptx::tma_load_3d(smem + Cfg::kK + st * Cfg::kTileBytes + c * kChunkBytes, &tk, &k_full[st], hk * HD + c * 64,
                           j * kBlk, b);
        if (!ptx::mbar_wait(&v_empty[st], ((j >> 1) & 1) ^ 1u, abort_flag)) break;
        ptx::mbar_expect_tx(&v_full[st], Cfg::kTileBytes);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          ptx::tma_load_3d(smem + Cfg::kV + st * Cfg::kTileBytes + c * kChunkBytes, &tv, &v_full[st], hk * HD + c * 64,
                           j * kBlk, b);
      }
    }
  } else if (warp == 1) {
    if (ptx::elect_one()) {
      const uint32_t idesc_s = ptx::make_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = ptx::make_idesc_bf16(128, HD, 0, 1);
      const uint32_t q_base = ptx::smem_u32(smem + Cfg::kQ);
      const uint32_t p_base = ptx::smem_u32(smem + Cfg::kP);
      const uint64_t q_desc = ptx::make_smem_desc(q_base, 16, 1024);
      const uint64_t k_desc0 = ptx::make_smem_desc(ptx::smem_u32(smem + Cfg::kK), 16, 1024);
      const uint64_t p_desc = ptx::make_smem_desc(p_base, 16, 1024);
      const uint64_t v_desc0 = ptx::make_smem_desc(ptx::smem_u32(smem + Cfg::kV), kChunkBytes, 1024);
      auto issue_s = [&](int j) {
        const uint64_t k_desc = desc_add(k_desc0, (j & 1) * Cfg::kTileBytes);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * kChunkBytes + (k & 3) * 32;
          ptx::mma_f16_ss(tS, desc_add(q_desc, off), desc_add(k_desc, off), idesc_s, k > 0);
        }
        ptx::tc_commit(s_full);
        ptx::tc_commit(&k_empty[j & 1]);   // the K tile may be refilled once this product has finished
      };
      bool ok = ptx::mbar_wait(q_full, 0, abort_flag) && ptx::mbar_wait(&k_full[0], 0, abort_flag);
      if (ok) {
        ptx::tc_fence_after_sync();
        issue_s(0);
      }
      for (int j = 0; j < nblk && ok; ++j) {
        if (j + 1 < nblk) {
          // S(j+1) goes into the score columns as soon as S(j) has been copied to registers
          if (!ptx::mbar_wait(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag)) break;
          if (!ptx::mbar_wait(s_free, j & 1, abort_flag)) break;
          ptx::tc_fence_after_sync();
          issue_s(j + 1);
        }
        if (!ptx::mbar_wait(&v_full[j & 1], (j >> 1) & 1, abort_flag)) break;
        if (!ptx::mbar_wait(p_full, j & 1, abort_flag)) break;
        ptx::tc_fence_after_sync();
        const uint64_t v_desc = desc_add(v_desc0, (j & 1) * Cfg::kTileBytes);
#pragma unroll
        for (int k = 0; k < kBlk / 16; ++k) {
          const uint32_t a_off = (k >> 2) * kChunkBytes + (k & 3) * 32;
          ptx::mma_f16_ss(tO, desc_add(p_desc, a_off), desc_add(v_desc, k * 2048), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
        }
        ptx::tc_commit(o_full);
        ptx::tc_commit(&v_empty[j & 1]);
      }
    }
  } else {
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int q_idx = q0 + row;
    const uint32_t lane_sel = static_cast<uint32_t>(quad * 32) << 16;
    const float sc = p.scale * kLog2e;
    constexpr float kLazy = 8.f;   // log2 of the largest P value tolerated before the reference maximum moves
    float m_ref = -INFINITY, l = 0.f;
    uint8_t* p_smem = smem + Cfg::kP;
    bool ok = true;
    for (int j = 0; j < nblk; ++j) {
      if (!ptx::mbar_wait_warp(s_full, j & 1, abort_flag)) { ok = false; break; }
      ptx::tc_fence_after_sync();
      uint32_t r0[32], r1[32], r2[32], r3[32];
      ptx::tmem_ld32(tS + lane_sel + 0, r0);
      ptx::tmem_ld32(tS + lane_sel + 32, r1);
      ptx::tmem_ld32(tS + lane_sel + 64, r2);
      ptx::tmem_ld32(tS + lane_sel + 96, r3);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(s_free);   // the score columns may be overwritten by S(j+1)
      const int kv0 = j * kBlk;
      if (j == qb) {  // diagonal block: keys after the query are masked
        const uint32_t ninf = __float_as_uint(-INFINITY);
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          if (kv0 + e > q_idx) r0[e] = ninf;
          if (kv0 + 32 + e > q_idx) r1[e] = ninf;
          if (kv0 + 64 + e > q_idx) r2[e] = ninf;
          if (kv0 + 96 + e > q_idx) r3[e] = ninf;
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        mx0 = max3(mx0, __uint_as_float(r0[e]), __uint_as_float(r0[e + 1]));
        mx1 = max3(mx1, __uint_as_float(r1[e]), __uint_as_float(r1[e + 1]));
        mx2 = max3(mx2, __uint_as_float(r2[e]), __uint_as_float(r2[e + 1]));
        mx3 = max3(mx3, __uint_as_float(r3[e]), __uint_as_float(r3[e + 1]));
      }
      const float m_blk = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * sc;
      bool waited_o = (j == 0);
      if (j == 0) {
        m_ref = m_blk;
      } else {
        const bool need = m_blk > m_ref + kLazy;
        if (__any_sync(0xffffffffu, need)) {
          // the previous P V product must have landed before O is rescaled in place
          if (!ptx::mbar_wait_warp(o_full, (j - 1) & 1, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after_sync();
          waited_o = true;
          const float alpha = need ? ex2(m_ref - m_blk) : 1.f;
#pragma unroll 1
          for (int c = 0; c < HD / 16; ++c) {
            uint32_t t[16];
            ptx::tmem_ld16(tO + lane_sel + c * 16, t);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) t[e] = __float_as_uint(__uint_as_float(t[e]) * alpha);
            ptx::tmem_st16(tO + lane_sel + c * 16, t);
          }
          ptx::tmem_st_wait();
          l *= alpha;
          if (need) m_ref = m_blk;
        }
      }
      const float neg = -m_ref;
      float rs0 = 0.f, rs1 = 0.f;
      auto exp_chunk = [&](uint32_t (&r)[32], int c) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float p0, p1;
          fma2(p0, p1, __uint_as_float(r[e]), __uint_as_float(r[e + 1]), sc, sc, neg, neg);
          p0 = ex2(p0);
          p1 = ex2(p1);
          add2(rs0, rs1, rs0, rs1, p0, p1);
          pk[e >> 1] = pack_bf16x2(p0, p1);
        }
        if (c == 0 && !waited_o) {
          // P(j-1) V(j-1) must have finished reading the P buffer before it is overwritten
          if (!ptx::mbar_wait_warp(o_full, (j - 1) & 1, abort_flag)) ok = false;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<uint4*>(p_smem + swz_off(row, c * 4 + u)) =
              make_uint4(pk[u * 4], pk[u * 4 + 1], pk[u * 4 + 2], pk[u * 4 + 3]);
      };
      exp_chunk(r0, 0);
      if (!ok) break;
      exp_chunk(r1, 1);
      exp_chunk(r2, 2);
      exp_chunk(r3, 3);
      l += rs0 + rs1;
      ptx::fence_proxy_async_smem();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(p_full);
    }
    if (ok) ok = ptx::mbar_wait_warp(o_full, (nblk - 1) & 1, abort_flag);
    if (ok) {
      ptx::tc_fence_after_sync();
      const float inv = 1.f / l;
      bf16* dst = p.o + (static_cast<long long>(b) * p.T + q_idx) * p.o_stride_t + h * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t r[32];
        ptx::tmem_ld32(tO + lane_sel + c * 32, r);
        ptx::tmem_ld_wait();
        if (q_idx < p.T) {
#pragma unroll
          for (int d = 0; d < 32; d += 8) {
            uint4 u;
            u.x = pack_bf16x2(__uint_as_float(r[d]) * inv, __uint_as_float(r[d + 1]) * inv);
            u.y = pack_bf16x2(__uint_as_float(r[d + 2]) * inv, __uint_as_float(r[d + 3]) * inv);
            u.z = pack_bf16x2(__uint_as_float(r[d + 4]) * inv, __uint_as_float(r[d + 5]) * inv);
            u.w = pack_bf16x2(__uint_as_float(r[d + 6]) * inv, __uint_as_float(r[d + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + d) = u;
          }
        }
      }
      if (q_idx < p.T)
        p.lse[(static_cast<long long>(b) * p.Hq + h) * p.T + q_idx] = (m_ref + log2f(l)) * 0.6931471805599453f;
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(p.status, kStatusMbarTimeout);
}

// ------------------------------------------------------------------------ backward
// Warps 0..7 element-wise, 8..11 dQ, 12 loads, 13 MMA issue.
constexpr int kBwdThreads = 448;

template <int HD>
struct BwdCfg {
  static constexpr int kTileBytes = kBlk * HD * 2;
  static constexpr bool kAlias = (HD == 128);       // tensor memory is full: P lies over S, dQ over dP
  static constexpr int kDoStages = (HD == 64) ? 2 : 1;
  static constexpr int kK = 0;
  static constexpr int kV = kK + kTileBytes;
  static constexpr int kQ = kV + kTileBytes;        // two stages
  static constexpr int kDO = kQ + 2 * kTileBytes;
  static constexpr int kDS = kDO + kDoStages * kTileBytes;
  static constexpr int kDQ = kDS + kBlk * kBlk * 2; // per dQ warp two [32 rows x 32 fp32] tiles that leave by TMA
  static constexpr int kStat = kDQ + 4 * 2 * 4096;  // per Q stage: 128 x (-lse log2 e), 128 x delta
  static constexpr int kBar = kStat + 2 * 2 * kBlk * 4;
  static constexpr int kSmem = kBar + 256;
  static constexpr int kTmemCols = 512;
  static constexpr int kColS = 0, kColDP = 128, kColDV = 256, kColDK = 256 + HD;
  static constexpr int kColDQ = kAlias ? kColDP : 384;
  // bf16 P, two queries per column: query half h starts at kColP + h * kPHalf
  static constexpr int kColP = kAlias ? kColS : 448;
  static constexpr int kPHalf = kAlias ? 64 : 32;
};

// Backward pipeline.  Scores are computed transposed (rows = keys, columns = queries), so that P^T can stay in tensor
// memory as the A operand of dV and only dS passes through shared memory, stored once and read as the K-major A operand
// of dK and as the MN-major A operand of dQ.  Per (query head, query block) iteration `it` the MMA warp issues
//     dV += P^T dO (it) | S^T = K Q^T (it+1) | dQ = dS K (it) | dK += dS^T Q (it) | dP^T = V dO^T (it+1)
// and the other warps work beside it:
//   element-wise warps: exponentials of it+1 under dQ, dK (it); dS of it+1 under dV (it+1), S (it+2).  Two warps share a
//     key row (query columns 0..63 and 64..127).  The row statistics of the queries are columns here; they come from
//     shared memory as broadcast reads.
//   dQ warps: copy dQ(it) out of tensor memory and add it to the fp32 accumulator by TMA reduce-adds of 32 x 32 tiles,
//     each warp on its own.
// MMAs execute in issue order, which orders most reuses: S(it+1) overwrites P(it) (hd 128) after dV(it) has read it, and
// dp_full(it+1) tells that dQ(it), dK(it) have read the dS buffer.
// Bound: at hd 128 the five products read 5 x 512 cycles of shared-memory operands an iteration, and dS, dQ and the loads
// move as much again; at hd 64 the 16384 exponentials take 1024 cycles and the products 1660.
// Measured (B200, with the delta and conversion passes; before = scores untransposed, P and dS through shared memory, dQ
// flushed by the element-wise warps): hd 128, 1 x 4096, 32 / 8 heads: 978 -> 351 us (980 TFLOP/s); hd 64, 4 x 2048,
// 32 / 8 heads: 376 -> 249 us; 8 x 1024, 12 heads: 117 -> 91 us; 3 x 777, 12 heads: 50 -> 32 us.
template <int HD>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                const __grid_constant__ CUtensorMap tdq, const AttnArgs p) {
  using Cfg = BwdCfg<HD>;
  constexpr int DS = Cfg::kDoStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kBar);
  uint64_t* kv_full = bars;            // 1
  uint64_t* q_full = bars + 1;         // [2]
  uint64_t* q_empty = bars + 3;        // [2]
  uint64_t* do_full = bars + 5;        // [2]
  uint64_t* do_empty = bars + 7;       // [2]
  uint64_t* stat_full = bars + 9;      // [2]  freed with the Q stage
  uint64_t* s_full = bars + 11;
  uint64_t* p_full = bars + 12;
  uint64_t* dp_full = bars + 13;
  uint64_t* ds_full = bars + 14;
  uint64_t* dq_full = bars + 15;
  uint64_t* dq_free = bars + 16;
  uint64_t* dkv_full = bars + 17;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;
  const int nqb = (p.T + kBlk - 1) / kBlk;
  // key block 0 meets every query block: the longest CTAs of all heads start first
  const int jb = blockIdx.y;
  const int hk = blockIdx.x % p.Hkv, b = blockIdx.x / p.Hkv;
  const int G = p.Hq / p.Hkv;
  const int nq = nqb - jb;     // query blocks jb .. nqb-1
  const int niter = G * nq;

  if (threadIdx.x == 0) {
    ptx::mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&q_full[s], 1); ptx::mbar_init(&q_empty[s], 1);
      ptx::mbar_init(&do_full[s], 1); ptx::mbar_init(&do_empty[s], 1);
      ptx::mbar_init(&stat_full[s], 1);
    }
    ptx::mbar_init(s_full, 1);
    ptx::mbar_init(p_full, 8);
    ptx::mbar_init(dp_full, 1);
    ptx::mbar_init(ds_full, 8);
    ptx::mbar_init(dq_full, 1);
    ptx::mbar_init(dq_free, 4);
    ptx::mbar_init(dkv_full, 1);
    *abort_flag = (ptx::smem_u32(smem) & 1023u) ? 1u : 0u;
    ptx::mbar_fence_init();
    ptx::tma_prefetch_desc(&tq);
    ptx::tma_prefetch_desc(&tk);
    ptx::tma_prefetch_desc(&tv);
    ptx::tma_prefetch_desc(&tdo);
    ptx::tma_prefetch_desc(&tdq);
  }
  if (warp == 13) {
    ptx::tmem_alloc(tmem_slot, Cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependency_wait();
  dependents_launch();
  const bool bad_align = (*abort_flag != 0);

  if (bad_align) {
    // fall through to the common exit
  } else if (warp == 12) {
    // ------------------------------------------------------------ loads
    const bool leader = ptx::elect_one();
    if (leader) {
      ptx::mbar_expect_tx(kv_full, 2 * Cfg::kTileBytes);
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) {
        ptx::tma_load_3d(smem + Cfg::kK + c * kChunkBytes, &tk, kv_full, hk * HD + c * 64, jb * kBlk, b);
        ptx::tma_load_3d(smem + Cfg::kV + c * kChunkBytes, &tv, kv_full, hk * HD + c * 64, jb * kBlk, b);
      }
    }
    bool ok = true;
    int it = 0;
    for (; it < niter; ++it) {
      const int g = it / nq, i = jb + (it - g * nq);
      const int h = hk * G + g;
      const int st = it & 1, dst = it % DS;
      // row statistics: requested before the waits; rows past the end of the sequence get lse = +inf, which turns their
      // probabilities into exact zeros
      float l[4], d[4];
      const float* lse_row = p.lse + (static_cast<long long>(b) * p.Hq + h) * p.T;
      const float* dlt_row = p.delta + (static_cast<long long>(b) * p.Hq + h) * p.T;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int q = i * kBlk + e * 32 + lane;
        l[e] = q < p.T ? lse_row[q] : INFINITY;
        d[e] = q < p.T ? dlt_row[q] : 0.f;
      }
      ok = ptx::mbar_wait(&q_empty[st], ((it >> 1) & 1) ^ 1u, abort_flag);
      if (__any_sync(0xffffffffu, !ok)) break;
      if (leader) {
        ptx::mbar_expect_tx(&q_full[st], Cfg::kTileBytes);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          ptx::tma_load_3d(smem + Cfg::kQ + st * Cfg::kTileBytes + c * kChunkBytes, &tq, &q_full[st], h * HD + c * 64,
                           i * kBlk, b);
      }
      float* stat = reinterpret_cast<float*>(smem + Cfg::kStat) + st * 2 * kBlk;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        stat[e * 32 + lane] = -l[e] * kLog2e;
        stat[kBlk + e * 32 + lane] = d[e];
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&stat_full[st]);
      ok = ptx::mbar_wait(&do_empty[dst], ((it / DS) & 1) ^ 1u, abort_flag);
      if (__any_sync(0xffffffffu, !ok)) break;
      if (leader) {
        ptx::mbar_expect_tx(&do_full[dst], Cfg::kTileBytes);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          ptx::tma_load_3d(smem + Cfg::kDO + dst * Cfg::kTileBytes + c * kChunkBytes, &tdo, &do_full[dst], h * HD + c * 64,
                           i * kBlk, b);
      }
    }
    if (it < niter && leader) {
      // gave up: copies already issued get a bounded chance to land before the CTA leaves
      const long long t0 = clock64();
      for (int s = 0; s < 5; ++s) {
        uint64_t* bar = s < 2 ? &q_full[s] : s < 4 ? &do_full[s - 2] : kv_full;
        while (!ptx::mbar_try_wait(bar, 0) && !ptx::mbar_try_wait(bar, 1) && clock64() - t0 < 4000000LL) {
        }
      }
    }
  } else if (warp == 13) {
    // ------------------------------------------------------------ MMA issue
    if (ptx::elect_one()) {
      const uint32_t idesc_s = ptx::make_idesc_bf16(128, 128, 0, 0);    // S^T, dP^T: K-major x K-major
      const uint32_t idesc_kv = ptx::make_idesc_bf16(128, HD, 0, 1);    // dV (A in tensor memory), dK: K-major x MN-major
      const uint32_t idesc_q = ptx::make_idesc_bf16(128, HD, 1, 1);     // dQ: MN-major x MN-major
      const uint32_t k_base = ptx::smem_u32(smem + Cfg::kK), v_base = ptx::smem_u32(smem + Cfg::kV);
      const uint32_t ds_base = ptx::smem_u32(smem + Cfg::kDS);
      const uint32_t q_base0 = ptx::smem_u32(smem + Cfg::kQ), do_base0 = ptx::smem_u32(smem + Cfg::kDO);
      const uint64_t k_kmaj = ptx::make_smem_desc(k_base, 16, 1024), v_kmaj = ptx::make_smem_desc(v_base, 16, 1024);
      const uint64_t k_mn = ptx::make_smem_desc(k_base, kChunkBytes, 1024);
      const uint64_t ds_kmaj = ptx::make_smem_desc(ds_base, 16, 1024), ds_mn = ptx::make_smem_desc(ds_base, kChunkBytes, 1024);
      const uint64_t q_kmaj0 = ptx::make_smem_desc(q_base0, 16, 1024), do_kmaj0 = ptx::make_smem_desc(do_base0, 16, 1024);
      const uint64_t q_mn0 = ptx::make_smem_desc(q_base0, kChunkBytes, 1024), do_mn0 = ptx::make_smem_desc(do_base0, kChunkBytes, 1024);
      auto issue_s = [&](int it) {
        const uint64_t q_d = desc_add(q_kmaj0, (it & 1) * Cfg::kTileBytes);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * kChunkBytes + (k & 3) * 32;
          ptx::mma_f16_ss(tmem_base + Cfg::kColS, desc_add(k_kmaj, off), desc_add(q_d, off), idesc_s, k > 0);
        }
        ptx::tc_commit(s_full);
      };
      auto issue_dp = [&](int it) {
        const uint64_t do_d = desc_add(do_kmaj0, (it % DS) * Cfg::kTileBytes);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * kChunkBytes + (k & 3) * 32;
          ptx::mma_f16_ss(tmem_base + Cfg::kColDP, desc_add(v_kmaj, off), desc_add(do_d, off), idesc_s, k > 0);
        }
        ptx::tc_commit(dp_full);
      };
      bool ok = ptx::mbar_wait(kv_full, 0, abort_flag) && ptx::mbar_wait(&q_full[0], 0, abort_flag);
      if (ok) {
        ptx::tc_fence_after_sync();
        issue_s(0);
        ok = ptx::mbar_wait(&do_full[0], 0, abort_flag);
      }
      if (ok) {
        ptx::tc_fence_after_sync();
        issue_dp(0);
      }
      for (int it = 0; it < niter && ok; ++it) {
        const uint64_t q_m = desc_add(q_mn0, (it & 1) * Cfg::kTileBytes), do_m = desc_add(do_mn0, (it % DS) * Cfg::kTileBytes);
        if (!ptx::mbar_wait(p_full, it & 1, abort_flag)) break;
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < kBlk / 16; ++k)  // reduction over the 128 queries
          ptx::mma_f16_ts(tmem_base + Cfg::kColDV, tmem_base + Cfg::kColP + (k >> 2) * Cfg::kPHalf + (k & 3) * 8,
                          desc_add(do_m, k * 2048), idesc_kv, (it > 0 || k > 0));
        ptx::tc_commit(&do_empty[it % DS]);
        if (it + 1 < niter) {
          if (!ptx::mbar_wait(&q_full[(it + 1) & 1], ((it + 1) >> 1) & 1, abort_flag)) break;
          ptx::tc_fence_after_sync();
          issue_s(it + 1);   // the scores of `it` were read before p_full(it)
        }
        if (!ptx::mbar_wait(ds_full, it & 1, abort_flag)) break;
        if (!Cfg::kAlias && it > 0 && !ptx::mbar_wait(dq_free, (it - 1) & 1, abort_flag)) break;
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int k = 0; k < kBlk / 16; ++k)  // reduction over the 128 keys
          ptx::mma_f16_ss(tmem_base + Cfg::kColDQ, desc_add(ds_mn, k * 2048), desc_add(k_mn, k * 2048), idesc_q, k > 0);
        ptx::tc_commit(dq_full);
#pragma unroll
        for (int k = 0; k < kBlk / 16; ++k)  // reduction over the 128 queries
          ptx::mma_f16_ss(tmem_base + Cfg::kColDK, desc_add(ds_kmaj, (k >> 2) * kChunkBytes + (k & 3) * 32),
                          desc_add(q_m, k * 2048), idesc_kv, (it > 0 || k > 0));
        ptx::tc_commit(&q_empty[it & 1]);
        if (it + 1 < niter) {
          if (!ptx::mbar_wait(&do_full[(it + 1) % DS], ((it + 1) / DS) & 1, abort_flag)) break;
          if (Cfg::kAlias && !ptx::mbar_wait(dq_free, it & 1, abort_flag)) break;
          ptx::tc_fence_after_sync();
          issue_dp(it + 1);
        } else {
          ptx::tc_commit(dkv_full);
        }
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------ dQ
    const int quad = warp & 3;
    const uint32_t t_dq = tmem_base + Cfg::kColDQ + (static_cast<uint32_t>(quad * 32) << 16);
    uint8_t* stg = smem + Cfg::kDQ + quad * 8192;
    auto stage = [&](const uint32_t (&r)[32], int piece) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<uint4*>(stg + piece * 4096 + lane * 128 + ((u ^ (lane & 7)) << 4)) =
            make_uint4(r[u * 4], r[u * 4 + 1], r[u * 4 + 2], r[u * 4 + 3]);
    };
    for (int it = 0; it < niter; ++it) {
      const int g = it / nq, i = jb + (it - g * nq);
      const int x = (hk * G + g) * HD, y = i * kBlk + quad * 32;
      if (!ptx::mbar_wait_warp(dq_full, it & 1, abort_flag)) break;
      ptx::tc_fence_after_sync();
      uint32_t r0[32], r1[32];
      ptx::tmem_ld32(t_dq, r0);
      ptx::tmem_ld32(t_dq + 32, r1);
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) {
        ptx::tmem_ld_wait();
        if (c == HD / 64 - 1) {
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(dq_free);       // the dQ columns may be overwritten
        }
        // the reduce-adds of the tiles staged before have finished reading them
        if (lane == 0) ptx::bulk_wait_read<0>();
        __syncwarp();
        stage(r0, 0);
        stage(r1, 1);
        if (c + 1 < HD / 64) {
          ptx::tmem_ld32(t_dq + (c + 1) * 64, r0);
          ptx::tmem_ld32(t_dq + (c + 1) * 64 + 32, r1);
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && y < p.T) {
#pragma unroll
          for (int h2 = 0; h2 < 2; ++h2)
            asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                             reinterpret_cast<uint64_t>(&tdq)),
                         "r"(ptx::smem_u32(stg + h2 * 4096)), "r"(x + c * 64 + h2 * 32), "r"(y), "r"(b)
                         : "memory");
          ptx::bulk_commit();
        }
      }
    }
    if (lane == 0) ptx::bulk_wait_all<0>();   // all reduce-adds done before the CTA exits
  } else {
    // ------------------------------------------------------------ element-wise
    const int quad = warp & 3, half = warp >> 2;
    const int row = quad * 32 + lane;                // key row
    const uint32_t lane_sel = static_cast<uint32_t>(quad * 32) << 16;
    const float sc = p.scale * kLog2e;
    const uint32_t tS = tmem_base + Cfg::kColS + lane_sel + half * 64, tDP = tmem_base + Cfg::kColDP + lane_sel + half * 64;
    const uint32_t tP = tmem_base + Cfg::kColP + lane_sel + half * Cfg::kPHalf;
    uint8_t* ds_row = smem + Cfg::kDS + half * kChunkBytes + row * 128;
    bool ok = true;
    for (int it = 0; it < niter; ++it) {
      const float* nl = reinterpret_cast<const float*>(smem + Cfg::kStat) + (it & 1) * 2 * kBlk + half * 64;
      const float* dl = nl + kBlk;
      if (!ptx::mbar_wait_warp(&stat_full[it & 1], (it >> 1) & 1, abort_flag)) { ok = false; break; }
      if (!ptx::mbar_wait_warp(s_full, it & 1, abort_flag)) { ok = false; break; }
      ptx::tc_fence_after_sync();
      uint32_t pr[2][32];
      ptx::tmem_ld32(tS, pr[0]);
      ptx::tmem_ld32(tS + 32, pr[1]);
      ptx::tmem_ld_wait();
      const bool diag = it % nq == 0;                // keys after the query get probability zero
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const float4 n4 = *reinterpret_cast<const float4*>(nl + c * 32 + e);
          float x0, x1, x2, x3;
          fma2(x0, x1, __uint_as_float(pr[c][e]), __uint_as_float(pr[c][e + 1]), sc, sc, n4.x, n4.y);
          fma2(x2, x3, __uint_as_float(pr[c][e + 2]), __uint_as_float(pr[c][e + 3]), sc, sc, n4.z, n4.w);
          x0 = ex2(x0); x1 = ex2(x1); x2 = ex2(x2); x3 = ex2(x3);
          if (diag) {
            const int q = half * 64 + c * 32 + e;
            if (row > q) x0 = 0.f;
            if (row > q + 1) x1 = 0.f;
            if (row > q + 2) x2 = 0.f;
            if (row > q + 3) x3 = 0.f;
          }
          pk[e / 2] = pack_bf16x2(x0, x1);
          pk[e / 2 + 1] = pack_bf16x2(x2, x3);
          pr[c][e] = __float_as_uint(x0); pr[c][e + 1] = __float_as_uint(x1);
          pr[c][e + 2] = __float_as_uint(x2); pr[c][e + 3] = __float_as_uint(x3);
        }
        ptx::tmem_st16(tP + c * 16, pk);
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(p_full);
      if (!ptx::mbar_wait_warp(dp_full, it & 1, abort_flag)) { ok = false; break; }
      ptx::tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t d[32];
        ptx::tmem_ld32(tDP + c * 32, d);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint32_t pk[4];
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const int e = u * 8 + v * 4;
            const float4 d4 = *reinterpret_cast<const float4*>(dl + c * 32 + e);
            float x0, x1, x2, x3;
            add2(x0, x1, __uint_as_float(d[e]), __uint_as_float(d[e + 1]), -d4.x, -d4.y);
            add2(x2, x3, __uint_as_float(d[e + 2]), __uint_as_float(d[e + 3]), -d4.z, -d4.w);
            mul2(x0, x1, x0, x1, __uint_as_float(pr[c][e]), __uint_as_float(pr[c][e + 1]));
            mul2(x2, x3, x2, x3, __uint_as_float(pr[c][e + 2]), __uint_as_float(pr[c][e + 3]));
            mul2(x0, x1, x0, x1, p.scale, p.scale);
            mul2(x2, x3, x2, x3, p.scale, p.scale);
            pk[v * 2] = pack_bf16x2(x0, x1);
            pk[v * 2 + 1] = pack_bf16x2(x2, x3);
          }
          *reinterpret_cast<uint4*>(ds_row + (((c * 4 + u) ^ (row & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
      ptx::fence_proxy_async_smem();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(ds_full);
    }
    if (ok) ok = ptx::mbar_wait_warp(dkv_full, 0, abort_flag);
    const int kv_idx = jb * kBlk + row;
    if (ok) {
      ptx::tc_fence_after_sync();
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        bf16* base = which == 0 ? p.dv : p.dk;
        const long long stride = which == 0 ? p.dv_stride_t : p.dk_stride_t;
        const uint32_t col = which == 0 ? Cfg::kColDV : Cfg::kColDK;
        bf16* dst = base + (static_cast<long long>(b) * p.T + kv_idx) * stride + hk * HD;
#pragma unroll 1
        for (int c = half * (HD / 64); c < (half + 1) * (HD / 64); ++c) {
          uint32_t r[32];
          ptx::tmem_ld32(tmem_base + col + lane_sel + c * 32, r);
          ptx::tmem_ld_wait();
          if (kv_idx < p.T) {
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
              uint4 u;
              u.x = pack_bf16x2(__uint_as_float(r[e]), __uint_as_float(r[e + 1]));
              u.y = pack_bf16x2(__uint_as_float(r[e + 2]), __uint_as_float(r[e + 3]));
              u.z = pack_bf16x2(__uint_as_float(r[e + 4]), __uint_as_float(r[e + 5]));
              u.w = pack_bf16x2(__uint_as_float(r[e + 6]), __uint_as_float(r[e + 7]));
              *reinterpret_cast<uint4*>(dst + c * 32 + e) = u;
            }
          }
        }
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 13) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(p.status, kStatusMbarTimeout);
}

// delta[b,h,t] = sum_d dO[b,t,h,d] * O[b,t,h,d], and the fp32 dQ accumulator starts at zero.  hd / 8 neighbouring lanes
// share a (b,t,h) row, 16 bytes of each operand per lane, so that every access of a warp is whole lines.
template <int HD>
__global__ void attn_delta_kernel(const bf16* __restrict__ d_o, const bf16* __restrict__ o, float* __restrict__ delta,
                                  float* __restrict__ dq_accum, int B, int T, int H, long long do_stride_t, long long o_stride_t) {
  dependents_launch();
  constexpr int L = HD / 8;
  const long long n = static_cast<long long>(B) * T * H * L;
  const long long n_up = (n + 31) / 32 * 32;   // whole warps take part in the shuffles
  for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < n_up; x += (long long)gridDim.x * blockDim.x) {
    const long long i = x / L;
    const int d = static_cast<int>(x % L) * 8;
    const int h = static_cast<int>(i % H);
    const long long bt = i / H;
    float s = 0.f;
    if (x < n) {
      const uint4 ua = *reinterpret_cast<const uint4*>(d_o + bt * do_stride_t + h * HD + d);
      const uint4 uc = *reinterpret_cast<const uint4*>(o + bt * o_stride_t + h * HD + d);
      const float2 a0 = unpack_bf16x2(ua.x), a1 = unpack_bf16x2(ua.y), a2 = unpack_bf16x2(ua.z), a3 = unpack_bf16x2(ua.w);
      const float2 c0 = unpack_bf16x2(uc.x), c1 = unpack_bf16x2(uc.y), c2 = unpack_bf16x2(uc.z), c3 = unpack_bf16x2(uc.w);
      s = a0.x * c0.x + a0.y * c0.y + a1.x * c1.x + a1.y * c1.y + a2.x * c2.x + a2.y * c2.y + a3.x * c3.x + a3.y * c3.y;
      float4* acc = reinterpret_cast<float4*>(dq_accum + i * HD + d);
      acc[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      acc[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int m = 1; m < L; m <<= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (d == 0 && x < n) {
      const long long b = bt / T, t = bt - b * T;
      delta[(b * H + h) * T + t] = s;
    }
  }
}

// dq (bf16, token stride dq_stride_t) = dq_accum (fp32 [B*T, H*hd])
__global__ void attn_dq_convert_kernel(const float* __restrict__ acc, bf16* __restrict__ dq, long long BT, int width,
                                       long long dq_stride_t) {
  dependents_launch();
  const int wv = width / 8;
  const long long n = BT * wv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long bt = i / wv;
    const int c = static_cast<int>(i - bt * wv) * 8;
    const float4 f0 = *reinterpret_cast<const float4*>(acc + bt * width + c);
    const float4 f1 = *reinterpret_cast<const float4*>(acc + bt * width + c + 4);
    uint4 u;
    u.x = pack_bf16x2(f0.x, f0.y); u.y = pack_bf16x2(f0.z, f0.w);
    u.z = pack_bf16x2(f1.x, f1.y); u.w = pack_bf16x2(f1.z, f1.w);
    *reinterpret_cast<uint4*>(dq + bt * dq_stride_t + c) = u;
  }
}

static bool attn_check(const TitbAttnDesc* d) {
  if (d->hd != 64 && d->hd != 128) return false;
  if (d->Hq % d->Hkv) return false;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (!al(d->q) || !al(d->k) || !al(d->v) || !al(d->o)) return false;
  if ((d->q_stride_t & 7) || (d->k_stride_t & 7) || (d->v_stride_t & 7) || (d->o_stride_t & 7)) return false;
  return true;
}

template <int HD>
static int attn_fwd_launch(const TitbAttnDesc* d, cudaStream_t st) {
  using Cfg = FwdCfg<HD>;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  // the maps end with a sequence: rows of the next one would meet probabilities of zero, which do not stop a NaN
  const uint64_t B = d->B, T = d->T, wq = static_cast<uint64_t>(d->Hq) * HD, wkv = static_cast<uint64_t>(d->Hkv) * HD;
  CUtensorMap tq, tk, tv;
  if (!make_tmap_tokens(&tq, d->q, 0, wq, T, B, d->q_stride_t, 64, kBlk) ||
      !make_tmap_tokens(&tk, d->k, 0, wkv, T, B, d->k_stride_t, 64, kBlk) ||
      !make_tmap_tokens(&tv, d->v, 0, wkv, T, B, d->v_stride_t, 64, kBlk))
    return TITB_ERR_TENSOR_MAP;
  AttnArgs a{};
  a.B = d->B; a.T = d->T; a.Hq = d->Hq; a.Hkv = d->Hkv; a.hd = HD;
  a.scale = d->scale;
  a.o = static_cast<bf16*>(d->o); a.lse = d->lse; a.o_stride_t = d->o_stride_t;
  a.status = titb_status_ptr();
  dim3 grid(static_cast<unsigned>(d->Hq) * d->B, (d->T + kBlk - 1) / kBlk);
  launch_dependent(attn_fwd_kernel<HD>, grid, kAttnThreads, Cfg::kSmem, st, tq, tk, tv, a);
  return static_cast<int>(cudaGetLastError());
}

template <int HD>
static int attn_bwd_launch(const TitbAttnDesc* d, cudaStream_t st) {
  using Cfg = BwdCfg<HD>;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  CUtensorMap tq, tk, tv, tdo, tdq;
  const uint64_t B = d->B, T = d->T, wq = static_cast<uint64_t>(d->Hq) * HD, wkv = static_cast<uint64_t>(d->Hkv) * HD;
  if (!make_tmap_tokens(&tq, d->q, 0, wq, T, B, d->q_stride_t, 64, kBlk) ||
      !make_tmap_tokens(&tk, d->k, 0, wkv, T, B, d->k_stride_t, 64, kBlk) ||
      !make_tmap_tokens(&tv, d->v, 0, wkv, T, B, d->v_stride_t, 64, kBlk) ||
      !make_tmap_tokens(&tdo, d->d_o, 0, wq, T, B, d->do_stride_t, 64, kBlk) ||
      !make_tmap_tokens(&tdq, d->dq_accum, 1, wq, T, B, wq, 32, 32))
    return TITB_ERR_TENSOR_MAP;
  const long long nrows = static_cast<long long>(d->B) * d->T * d->Hq;
  const long long delta_blocks = (nrows * (HD / 8) + 255) / 256, delta_max = device_sm_count() * 16LL;
  attn_delta_kernel<HD><<<static_cast<int>(delta_blocks < delta_max ? delta_blocks : delta_max), 256, 0, st>>>(
      static_cast<const bf16*>(d->d_o), static_cast<const bf16*>(d->o), d->delta, d->dq_accum, d->B, d->T, d->Hq,
      d->do_stride_t, d->o_stride_t);
  AttnArgs a{};
  a.B = d->B; a.T = d->T; a.Hq = d->Hq; a.Hkv = d->Hkv; a.hd = HD;
  a.scale = d->scale;
  a.lse = d->lse; a.delta = d->delta; a.dq_accum = d->dq_accum;
  a.dk = static_cast<bf16*>(d->dk); a.dv = static_cast<bf16*>(d->dv);
  a.dk_stride_t = d->dk_stride_t; a.dv_stride_t = d->dv_stride_t;
  a.status = titb_status_ptr();
  dim3 grid(static_cast<unsigned>(d->Hkv) * d->B, (d->T + kBlk - 1) / kBlk);
  launch_dependent(attn_bwd_kernel<HD>, grid, kBwdThreads, Cfg::kSmem, st, tq, tk, tv, tdo, tdq, a);
  const long long bt = static_cast<long long>(d->B) * d->T;
  const int width = d->Hq * HD;
  int cb = static_cast<int>((bt * (width / 8) + 255) / 256);
  if (cb > device_sm_count() * 8) cb = device_sm_count() * 8;
  attn_dq_convert_kernel<<<cb, 256, 0, st>>>(d->dq_accum, static_cast<bf16*>(d->dq), bt, width, d->dq_stride_t);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace titb

using namespace titb;

TITB_API int titb_attn_fwd(const TitbAttnDesc* d, cudaStream_t stream) {
  (void)cudaGetLastError();
  if (d->B <= 0 || d->T <= 0) return 0;
  if (!attn_check(d)) return TITB_ERR_SHAPE;
  return d->hd == 64 ? attn_fwd_launch<64>(d, stream) : attn_fwd_launch<128>(d, stream);
}

TITB_API int titb_attn_bwd(const TitbAttnDesc* d, cudaStream_t stream) {
  (void)cudaGetLastError();
  if (d->B <= 0 || d->T <= 0) return 0;
  if (!attn_check(d)) return TITB_ERR_SHAPE;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (!al(d->d_o) || !al(d->dq) || !al(d->dk) || !al(d->dv) || (d->do_stride_t & 7) || (d->dq_stride_t & 7) ||
      (d->dk_stride_t & 7) || (d->dv_stride_t & 7))
    return TITB_ERR_ALIGNMENT;
  return d->hd == 64 ? attn_bwd_launch<64>(d, stream) : attn_bwd_launch<128>(d, stream);
}
