// fp32 GEMM on the 5th-generation tensor cores, at fp32 accuracy.
//
// Counterpart of the reference's cublasSgemm call sites (infini_train/src/kernels/cuda/linear.cu:26-47 Matmul,
// :103-126 LinearForward, :172-229 LinearBackward) for fp32 tensors.
//
// An fp32 value is the exact sum of three bf16 values (8 + 8 + 8 significant bits): x = x0 + x1 + x2 with x0 = bf16(x),
// x1 = bf16(x - x0), x2 = x - x0 - x1.  A product a b is then
//     a0 b0 + (a0 b1 + a1 b0) + (a0 b2 + a1 b1 + a2 b0)  +  terms below 2^-25 |a b|
// -- six bf16 products, each exact in the tensor core's fp32 accumulator, whose omitted rest is smaller than the rounding
// of one fp32 product.  The tensor core truncates when it adds, so it only accumulates over 64 reduction steps, the small
// products first; those 64-step partial sums are read out of tensor memory and added in registers with round-to-nearest.
// Against float64 the result is as close as the sequential fp32 FMA chain it replaces, or closer
// (tests/test_gpu_sgemm.py holds it to that).
//
// The range is that of fp32.  x1 and x2 are stored 2^15 times as large, so that they do not fall under the smallest bf16
// (without it a value below 2^-110 loses bits), and the sum is scaled back by the first MMA of the product that follows.
// Values below 2^-125 count to within 2^-148, the two last bits of a subnormal number.  At the upper end bf16(x) is infinite
// from 2^128 (1 - 2^-9) on, inf - inf appears inside the split of an infinity, and scaled parts or products may overflow where
// x (from 2^120 on) or the sum (from about 2^114 on) does not.  All of these, and NaN operands, leave a non-finite sum.  A warp
// that finds one leaves its 32 x 64 piece of the tile out, and when the CTA is through its tiles it computes such pieces again
// as a chain of fp32 multiply-adds, which gives IEEE's answer (finfo.min as a mask, infinities).  2048 x 3072 x 768 with one
// infinity: 276 us, with nothing but NaNs: 652 us, against 87 us of finite operands and 480 us of the kernel before.
//
// Bound: the six products are 6 x 2 M N K tensor FLOPs, i.e. 278 TFLOP/s of fp32 work at the measured bf16 peak, about four
// times what 148 SMs x 128 FMA lanes can do.  One CTA works on a 128 x 128 tile:
//   warps 0..7   read the fp32 tiles (K- or MN-major, as they lie in memory) a chunk ahead into registers, split them and
//                write six swizzled bf16 tiles (3 x 16 KB per operand) of a two-stage ring
//   warps 8..15  add the accumulator of every 64-deep chunk to 64 registers per thread, and store the tile
//   warp 16      issues 4 x 6 tcgen05.mma 128 x 128 x 16 per chunk; two accumulators alternate
// Splitting in the kernel costs about 1000 issue slots per chunk and scheduler, under the 1536 cycles of its MMAs; a
// separate split pass would write and read another 6 bytes per element.
// Measured (B200, GPT-2 124M layers, forward / input gradient / weight gradient), before = a 64 x 64 CUDA-core kernel:
//   2048 tokens, 3072 x 768:  473 / 669 / 698 us before,  86 / 105 / 76 us now (112 / 92 / 127 TFLOP/s)
//   2048 tokens, 50304 x 768: 7.1 / 11.6 / 10.6 ms before, 1.06 / 1.53 / 1.11 ms now
//   128 tokens,  50304 x 768: 511 / 8908 / 685 us before,  92 / 213 / 102 us now
//   rms error against float64 at K = 768: 5.0e-7 before, 1.0e-7 now; at K = 50304: 4.0e-6 before, 2e-7 to 5e-7 now
// Few output tiles (small batches, long reductions): a cluster of 2, 4 or 8 CTAs shares one tile's reduction, and the
// partial tiles are summed through distributed shared memory in a fixed order -- no workspace, no atomics.  Very short
// reductions: sgemm_short_kernel.
#include <cuda.h>
#include <cuda_runtime.h>
#include <limits.h>

#include "api.h"
#include "ptx_sm100.cuh"

namespace titb {

namespace {

constexpr int kST = 128;                 // tile rows and columns
constexpr int kSK = 64;                  // reduction chunk
constexpr int kPlane = kST * kSK * 2;    // one bf16 tile of one operand part: 16 KB
constexpr int kOperand = 3 * kPlane;
constexpr int kSStage = 2 * kOperand;    // A and B parts: 96 KB
constexpr int kSStages = 2;
constexpr int kPartShift = 15;           // the second and third part of a value are stored 2^15 times as large (the most an MMA scales)
constexpr float kPartScale = 1 << kPartShift;
constexpr int kConvWarps = 8, kDrainWarps = 8;
constexpr int kSThreads = (kConvWarps + kDrainWarps + 1) * 32;
constexpr int kRedStride = kST + 4;      // floats per row of the partial tile in shared memory (conflict-free 16-byte rows)
constexpr int kSlabK = 16;               // reduction steps that fma_tile stages at a time, behind the partial tile
constexpr int kSSmem = kSStages * kSStage + 1024 /*alignment slack*/ + 256 /*barriers, pieces left out*/;
static_assert((kST + 2 * kSlabK) * kRedStride * 4 <= kSStages * kSStage, "the partial tile and the slabs reuse the operand ring");

struct SgemmArgs {
  const float *a, *b;
  float* c;
  int M, N, K;
  int a_mn, b_mn;        // operand stored [K, rows] instead of [rows, K]
  long long lda, ldb;
  int a_vec, b_vec;      // 16-byte loads allowed
  int c_vec;             // 32-byte stores allowed
  int accumulate;
  int split;             // CTAs of the cluster that share one tile
  int chunks_per_cta;
  int* status;
};

// Eight consecutive values of one operand: `line` runs over the strided direction, `c` over the contiguous one.
__device__ __forceinline__ void load_unit(float (&v)[8], const float* base, long long ld, long long line, int nlines, int c,
                                          int extent, int vec) {
  if (line < nlines && c + 8 <= extent && vec) {
    const float4* p = reinterpret_cast<const float4*>(base + line * ld + c);
    const float4 x = __ldg(p), y = __ldg(p + 1);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = (line < nlines && c + e < extent) ? __ldg(base + line * ld + c + e) : 0.f;
  }
}

// Splits eight values into their three bf16 parts, the second and the third times kPartScale, and stores each part's 16
// bytes.  The differences and the scaling are exact.
__device__ __forceinline__ void split_store(const float (&v)[8], uint8_t* dst) {
  uint32_t p0[4], p1[4], p2[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float x = v[2 * e], y = v[2 * e + 1];
    p0[e] = pack_bf16x2(x, y);
    fma2(x, y, __uint_as_float(p0[e] << 16), __uint_as_float(p0[e] & 0xffff0000u), -1.f, -1.f, x, y);
    mul2(x, y, x, y, kPartScale, kPartScale);
    p1[e] = pack_bf16x2(x, y);
    fma2(x, y, __uint_as_float(p1[e] << 16), __uint_as_float(p1[e] & 0xffff0000u), -1.f, -1.f, x, y);
    p2[e] = pack_bf16x2(x, y);
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(p0[0], p0[1], p0[2], p0[3]);
  *reinterpret_cast<uint4*>(dst + kPlane) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
  *reinterpret_cast<uint4*>(dst + 2 * kPlane) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n\t}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}

// Pieces that the warps which sum the chunks left out: bit n of `tiles` for the CTA's n-th tile, and from tile number `from` on
// every piece (set by the first one that has no bit).
struct Redo {
  uint32_t tiles[kDrainWarps];
  int from[kDrainWarps];
  __device__ void clear(int w) {
    tiles[w] = 0;
    from[w] = INT_MAX;
  }
  __device__ bool any(int w) const { return tiles[w] || from[w] != INT_MAX; }
  __device__ void leave_out(int w, int tile, int first, int step) {
    const int n = (tile - first) / step;
    if (n < 32) tiles[w] |= 1u << n;
    else from[w] = min(from[w], tile);
  }
  __device__ bool left_out(int w, int tile, int first, int step) const {
    if (!any(w)) return false;
    const int n = (tile - first) / step;
    return tile >= from[w] || (n < 32 && (tiles[w] >> n & 1u));
  }
};

// Computes one tile over k0 <= k < k1 on the CUDA cores, one rounding per step in ascending order, and hands the values of the
// pieces in the mask `pieces` to put(row, column, value).  The whole CTA calls it; 512 threads hold 8 x 4 values each.  It comes
// after the tile loop so that its registers are not the tile loop's: in the loop, it made every call 8 % slower.
template <typename Put>
__device__ __forceinline__ void fma_tile(const SgemmArgs& p, int m0, int n0, int k0, int k1, uint32_t pieces, float* slab, Put put) {
  float* as = slab;
  float* bs = slab + kSlabK * kRedStride;
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const bool work = tid < 512;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  // element e of a slab: neighbouring threads read along the contiguous direction of the operand
  auto fill = [&](float* dst, const float* base, long long ld, int mn, int r0, int rows, int k) {
#pragma unroll
    for (int i = 0; i < kSlabK * kST / 512; ++i) {
      const int e = i * 512 + tid;
      const int s = mn ? e / kST : e % kSlabK, r = mn ? e % kST : e / kSlabK;
      const bool in = k + s < k1 && r0 + r < rows;
      dst[s * kRedStride + r] = in ? __ldg(base + (mn ? (k + s) * ld + r0 + r : (r0 + r) * ld + k + s)) : 0.f;
    }
  };
#pragma unroll 1
  for (int k = k0; k < k1; k += kSlabK) {
    __syncthreads();   // the slabs before have been read
    if (work) {
      fill(as, p.a, p.lda, p.a_mn, m0, p.M, k);
      fill(bs, p.b, p.ldb, p.b_mn, n0, p.N, k);
    }
    __syncthreads();
    if (work) {
#pragma unroll 1
      for (int s = 0; s < kSlabK; ++s) {
        float x[8], y[4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float4*>(x + 4 * h) = *reinterpret_cast<const float4*>(as + s * kRedStride + h * 64 + ty * 4);
        *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(bs + s * kRedStride + tx * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
      }
    }
  }
  if (!work) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = (i >> 2) * 64 + ty * 4 + (i & 3);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tx * 4 + j;
      if (pieces >> ((c >> 6) * 4 + (r >> 5)) & 1u) put(r, c, acc[i][j]);
    }
  }
}

__global__ void __launch_bounds__(kSThreads, 1) sgemm_split3_kernel(const SgemmArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kSStages * kSStage);
  uint64_t* empty = full + kSStages;
  uint64_t* acc_full = empty + kSStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  Redo* redo = reinterpret_cast<Redo*>(smem + kSStages * kSStage + 128);
  const int warp = ptx::warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kSStages; ++s) {
      ptx::mbar_init(&full[s], kConvWarps);
      ptx::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&acc_full[b], 1);
      ptx::mbar_init(&acc_empty[b], kDrainWarps);
    }
    *abort_flag = 0;
    for (int w = 0; w < kDrainWarps; ++w) redo->clear(w);
    ptx::mbar_fence_init();
  }
  if (warp == kConvWarps + kDrainWarps) {
    ptx::tmem_alloc(tmem_slot, 2 * kST);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependency_wait();
  dependents_launch();

  const int tiles_m = (p.M + kST - 1) / kST, tiles_n = (p.N + kST - 1) / kST;
  const int tiles = tiles_m * tiles_n;
  const int nchunk = (p.K + kSK - 1) / kSK;
  // CTAs of a cluster have neighbouring block indices; a cluster works on one tile (split == 1: CTAs walk the tiles)
  const int part = static_cast<int>(blockIdx.x) % p.split;
  const int first = static_cast<int>(blockIdx.x) / p.split, step = static_cast<int>(gridDim.x) / p.split;
  const int c0 = part * p.chunks_per_cta, c1 = min(nchunk, c0 + p.chunks_per_cta);
  const int per_tile = max(0, c1 - c0);

  if (warp < kConvWarps) {
    // ------------------------------------------------- read, split, store
    const int tid = threadIdx.x, u = tid & 7, l0 = tid >> 3;
    float va[4][8], vb[4][8];
    // a line of shared memory is 64 consecutive values: of K for one row (K-major), or of 64 rows for one k (MN-major)
    auto load = [&](float (&v)[4][8], const float* base, long long ld, int mn, int rows, int r0, int k0, int vec) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int l = l0 + 32 * i;
        if (!mn) load_unit(v[i], base, ld, r0 + l, rows, k0 + u * 8, p.K, vec);
        else load_unit(v[i], base, ld, k0 + (l & 63), p.K, r0 + (l & 64) + u * 8, rows, vec);
      }
    };
    auto load_chunk = [&](int tile, int c) {
      load(va, p.a, p.lda, p.a_mn, p.M, (tile % tiles_m) * kST, c * kSK, p.a_vec);
      load(vb, p.b, p.ldb, p.b_mn, p.N, (tile / tiles_m) * kST, c * kSK, p.b_vec);
    };
    int stage = 0;
    uint32_t phase = 0;
    int tile = first, c = c0;
    bool more = tile < tiles && per_tile > 0;
    if (more) load_chunk(tile, c);
    while (more) {
      if (!ptx::mbar_wait_warp(&empty[stage], phase ^ 1u, abort_flag)) break;
      uint8_t* dst = smem + stage * kSStage;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int l = l0 + 32 * i;
        const uint32_t off = static_cast<uint32_t>(l * 128 + ((u ^ (l & 7)) << 4));
        split_store(va[i], dst + off);
        split_store(vb[i], dst + kOperand + off);
      }
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&full[stage]);
      if (++stage == kSStages) { stage = 0; phase ^= 1u; }
      if (++c == c1) {
        c = c0;
        tile += step;
        more = tile < tiles;
      }
      if (more) load_chunk(tile, c);
    }
  } else if (warp == kConvWarps + kDrainWarps) {
    // ------------------------------------------------- MMA issuer
    if (ptx::elect_one()) {
      const uint32_t idesc = ptx::make_idesc_bf16(kST, kST, p.a_mn, p.b_mn);
      const uint32_t a_lbo = p.a_mn ? 64 * kSK * 2 : 16, b_lbo = p.b_mn ? 64 * kSK * 2 : 16;
      const uint32_t a_step = p.a_mn ? 16 * 128 : 32, b_step = p.b_mn ? 16 * 128 : 32;
      // smallest products first; {part of A, part of B}; the first is 2^30 times as large, the last as it is, the
      // others 2^15 times
      constexpr int kPa[6] = {1, 0, 2, 0, 1, 0}, kPb[6] = {1, 2, 0, 1, 0, 0};
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step) {
        for (int c = 0; c < per_tile; ++c, ++it) {
          const int buf = it & 1;
          if (!ptx::mbar_wait(&acc_empty[buf], ((it >> 1) & 1) ^ 1u, abort_flag) ||
              !ptx::mbar_wait(&full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t sa = ptx::smem_u32(smem + stage * kSStage), sb = sa + kOperand;
          const uint32_t d = tmem_base + buf * kST;
#pragma unroll
          for (int q = 0; q < 6; ++q) {
            const uint64_t ad = ptx::make_smem_desc(sa + kPa[q] * kPlane, a_lbo, 1024);
            const uint64_t bd = ptx::make_smem_desc(sb + kPb[q] * kPlane, b_lbo, 1024);
#pragma unroll
            for (int k = 0; k < kSK / 16; ++k) {   // only the address field of the descriptors moves
              const uint64_t ak = ad + ((k * a_step) >> 4), bk = bd + ((k * b_step) >> 4);
              if (k == 0 && (q == 1 || q == 5)) ptx::mma_f16_ss_scaled<kPartShift>(d, ak, bk, idesc);
              else ptx::mma_f16_ss(d, ak, bk, idesc, (q > 0 || k > 0) ? 1u : 0u);
            }
          }
          ptx::tc_commit(&empty[stage]);
          ptx::tc_commit(&acc_full[buf]);
          if (++stage == kSStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else {
    // ------------------------------------------------- sum the chunks, store the tile
    const int quad = warp & 3, half = (warp - kConvWarps) >> 2;
    const int row = quad * 32 + lane;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * 64;
    int it = 0;
    bool ok = true;
    for (int tile = first; tile < tiles && ok; tile += step) {
      float acc[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = 0.f;
      for (int c = 0; c < per_tile; ++c, ++it) {
        const int buf = it & 1;
        if (!ptx::mbar_wait_warp(&acc_full[buf], (it >> 1) & 1, abort_flag)) { ok = false; break; }
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t r[16];
          ptx::tmem_ld16(t_row + buf * kST + g * 16, r);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[g * 16 + j] += __uint_as_float(r[j]);
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&acc_empty[buf]);
      }
      if (!ok) break;
      const int gr = (tile % tiles_m) * kST + row, gc = (tile / tiles_m) * kST + half * 64;
      float finite = 0.f;
#pragma unroll
      for (int j = 0; j < 64; ++j) finite = fmaf(acc[j], 0.f, finite);
      // (kept in shared memory: in registers this made the whole kernel spill)
      if (gc < p.N && __any_sync(0xffffffffu, !(finite == 0.f)) && lane == 0) redo->leave_out(warp - kConvWarps, tile, first, step);
      __syncwarp();
      if (redo->left_out(warp - kConvWarps, tile, first, step)) continue;   // a cluster works on one tile: ends its loop
      if (p.split > 1) {
        // every MMA of this CTA has finished (the last accumulator was read), so the operand ring is free
        float* red = reinterpret_cast<float*>(smem) + row * kRedStride + half * 64;
#pragma unroll
        for (int j = 0; j < 64; j += 4)
          *reinterpret_cast<float4*>(red + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        break;
      }
      if (gr < p.M && gc < p.N) {
        float* out = p.c + static_cast<long long>(gr) * p.N + gc;
        if (p.c_vec && gc + 64 <= p.N) {
#pragma unroll
          for (int j = 0; j < 64; j += 8) {
            if (p.accumulate) {
              const float4 x = *reinterpret_cast<const float4*>(out + j), y = *reinterpret_cast<const float4*>(out + j + 4);
              acc[j] += x.x; acc[j + 1] += x.y; acc[j + 2] += x.z; acc[j + 3] += x.w;
              acc[j + 4] += y.x; acc[j + 5] += y.y; acc[j + 6] += y.z; acc[j + 7] += y.w;
            }
            // a thread owns a row piece: 32-byte stores fill whole sectors
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + j), "f"(acc[j]), "f"(acc[j + 1]),
                         "f"(acc[j + 2]), "f"(acc[j + 3]), "f"(acc[j + 4]), "f"(acc[j + 5]), "f"(acc[j + 6]), "f"(acc[j + 7])
                         : "memory");
          }
        } else {
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (gc + j < p.N) out[j] = p.accumulate ? out[j] + acc[j] : acc[j];
        }
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncwarp();   // the lanes of the MMA warp meet again
  __syncthreads();
  bool again = false;
  for (int w = 0; w < kDrainWarps; ++w) again |= redo->any(w);
  if (again && !*abort_flag) {
    float* red = reinterpret_cast<float*>(smem);
    for (int tile = first; tile < tiles; tile += step) {
      uint32_t pieces = 0;
      for (int w = 0; w < kDrainWarps; ++w) pieces |= static_cast<uint32_t>(redo->left_out(w, tile, first, step)) << w;
      if (!pieces) continue;
      const int m0 = (tile % tiles_m) * kST, n0 = (tile / tiles_m) * kST;
      fma_tile(p, m0, n0, c0 * kSK, min(p.K, c1 * kSK), pieces, red + kST * kRedStride, [&](int r, int c, float v) {
        if (p.split > 1) {
          red[r * kRedStride + c] = v;
        } else if (m0 + r < p.M && n0 + c < p.N) {
          float* out = p.c + static_cast<long long>(m0 + r) * p.N + n0 + c;
          *out = p.accumulate ? *out + v : v;
        }
      });
    }
  }
  if (p.split > 1) {
    ptx::cluster_sync_all();   // every CTA's partial tile is in its shared memory
    const int rows = kST / p.split, tile = first;
    const uint32_t base = ptx::smem_u32(smem);
    for (int i = threadIdx.x; i < rows * (kST / 4); i += kSThreads) {
      const int row = part * rows + i / (kST / 4), col = (i % (kST / 4)) * 4;
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r = 0; r < p.split; ++r) {
        const float4 v = ld_cluster_f4(base + (row * kRedStride + col) * 4, r);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      const int gr = (tile % tiles_m) * kST + row, gc = (tile / tiles_m) * kST + col;
      if (gr < p.M && gc < p.N) {
        float* out = p.c + static_cast<long long>(gr) * p.N + gc;
        if (p.c_vec && gc + 4 <= p.N) {
          float4* o = reinterpret_cast<float4*>(out);
          if (p.accumulate) {
            const float4 v = *o;
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
          }
          *o = s;
        } else {
          const float sv[4] = {s.x, s.y, s.z, s.w};
          for (int j = 0; j < 4 && gc + j < p.N; ++j) out[j] = p.accumulate ? out[j] + sv[j] : sv[j];
        }
      }
    }
    ptx::cluster_sync_all();   // nobody leaves while its shared memory is being read
  }
  if (warp == kConvWarps + kDrainWarps) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, 2 * kST);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(p.status, kStatusMbarTimeout);
}

// Reductions of at most KM steps: a 64 x 64 tile per CTA on the CUDA cores, the whole reduction loaded at once, 4 x 4 values per
// thread, one rounding per step in ascending order.  A chunk of the kernel above is 64 steps deep, and its set-up (barriers,
// tensor memory, two hand-overs between warps) takes longer than such a product.  Measured (B200, us, K = 16 / 32, the kernel
// above -> this one): 16 x 16 7.1 -> 2.1 / 7.1 -> 3.1, 1024 x 1024 8.1 -> 3.2 / 8.1 -> 4.8, 2048 x 2048 12.8 -> 7.2 / 12.9 -> 12.2,
// 4096 x 4096 34.6 -> 24.3 / 34.8 -> 42.0.
template <int KM>
__global__ void __launch_bounds__(256) sgemm_short_kernel(const SgemmArgs p) {
  dependency_wait();
  dependents_launch();
  __shared__ float4 as[KM][17], bs[KM][17];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int tiles_m = (p.M + 63) / 64;
  const int m0 = static_cast<int>(blockIdx.x % tiles_m) * 64, n0 = static_cast<int>(blockIdx.x / tiles_m) * 64;
  float va[KM / 4], vb[KM / 4];
  // neighbouring threads read along the contiguous direction of the operand
  auto at = [&](int i, int mn, int& k, int& r) {
    const int e = i * 256 + tid;
    k = mn ? e >> 6 : e % KM;
    r = mn ? e & 63 : e / KM;
  };
  auto load = [&](float (&v)[KM / 4], const float* base, long long ld, int mn, int r0, int rows) {
#pragma unroll
    for (int i = 0; i < KM / 4; ++i) {
      int k, r;
      at(i, mn, k, r);
      v[i] = k < p.K && r0 + r < rows ? __ldg(base + (mn ? k * ld + r0 + r : (r0 + r) * ld + k)) : 0.f;
    }
  };
  auto store = [&](const float (&v)[KM / 4], float4 (&dst)[KM][17], int mn) {
#pragma unroll
    for (int i = 0; i < KM / 4; ++i) {
      int k, r;
      at(i, mn, k, r);
      reinterpret_cast<float*>(dst[k])[r] = v[i];
    }
  };
  load(va, p.a, p.lda, p.a_mn, m0, p.M);
  load(vb, p.b, p.ldb, p.b_mn, n0, p.N);
  store(va, as, p.a_mn);
  store(vb, bs, p.b_mn);
  __syncthreads();
  float acc[4][4] = {};
#pragma unroll 8
  for (int k = 0; k < p.K; ++k) {
    const float4 x = as[k][ty], y = bs[k][tx];
    const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xs[i], ys[j], acc[i][j]);
  }
  const int c = n0 + tx * 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = m0 + ty * 4 + i;
    if (r >= p.M) break;
    float* out = p.c + static_cast<long long>(r) * p.N + c;
    if (p.c_vec && c + 4 <= p.N) {
      float4* o = reinterpret_cast<float4*>(out);
      float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      if (p.accumulate) {
        const float4 old = *o;
        v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
      }
      *o = v;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < p.N) out[j] = p.accumulate ? out[j] + acc[i][j] : acc[i][j];
    }
  }
}

// CTAs per tile: the fewest rounds of chunks on the busiest SM, with a charge for the exchange of the partial tiles (about
// three chunks).  Parts are whole multiples of ceil(chunks / parts): the last ones may have nothing to add but zeros (nine
// chunks over eight parts), which costs nothing, as the others take no longer for it.  That all clusters run at the same time
// is assumed, not asked: clusters of eight may wait for room within a group of SMs.
int pick_split(int tiles, int nchunk, int sms) {
  int best = 1;
  double cost = 1e30;
  for (int s = 1; s <= 8; s *= 2) {
    if (s > 1 && (s > nchunk || tiles * s > sms)) break;
    const double waves = s > 1 ? 1.0 : static_cast<double>((tiles + sms - 1) / sms);
    const double c = waves * ((nchunk + s - 1) / s) + (s > 1 ? 3.0 : 0.0);
    if (c < cost) { cost = c; best = s; }
  }
  return best;
}

}  // namespace
}  // namespace titb

using namespace titb;

TITB_API int titb_sgemm(const float* A, const float* B, float* C, int M, int N, int K, int trans_a, int trans_b,
                        int accumulate, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  (void)cudaGetLastError();
  if (K <= 0)
    return accumulate ? 0 : static_cast<int>(cudaMemsetAsync(C, 0, sizeof(float) * static_cast<size_t>(M) * N, stream));
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  SgemmArgs a{};
  a.a = A; a.b = B; a.c = C;
  a.M = M; a.N = N; a.K = K;
  a.a_mn = trans_a ? 1 : 0;
  a.b_mn = trans_b ? 0 : 1;      // op(B) = B^T means B is stored [N, K]
  a.lda = trans_a ? M : K;
  a.ldb = trans_b ? K : N;
  a.accumulate = accumulate;
  a.c_vec = (reinterpret_cast<uintptr_t>(C) & 31) == 0 && !(N & 7);
  // where the lines lie: see sgemm_short_kernel
  if (K <= 16 || (K <= 32 && static_cast<long long>(M) * N <= 1 << 22)) {
    const cudaError_t e = launch_dependent(K <= 16 ? sgemm_short_kernel<16> : sgemm_short_kernel<32>,
                                           static_cast<unsigned>(((M + 63) / 64) * ((N + 63) / 64)), 256, 0, stream, a);
    return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
  }
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(sgemm_split3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  a.a_vec = al16(A) && !(a.lda & 3);
  a.b_vec = al16(B) && !(a.ldb & 3);
  a.status = titb_status_ptr();
  if (!a.status) return static_cast<int>(cudaErrorMemoryAllocation);
  const int sms = device_sm_count();
  const int tiles = ((M + kST - 1) / kST) * ((N + kST - 1) / kST), nchunk = (K + kSK - 1) / kSK;
  a.split = pick_split(tiles, nchunk, sms);
  a.chunks_per_cta = (nchunk + a.split - 1) / a.split;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.split > 1 ? tiles * a.split : (tiles < sms ? tiles : sms));
  cfg.blockDim = dim3(kSThreads);
  cfg.dynamicSmemBytes = kSSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = a.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, sgemm_split3_kernel, a);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}
