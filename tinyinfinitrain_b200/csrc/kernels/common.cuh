// Shared device helpers for the sm_100a kernel set: 128-bit vector IO, bf16
// packing, warp/block reductions and the error-status convention.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace titb {

using bf16 = __nv_bfloat16;
using bf162 = __nv_bfloat162;

// Error codes written to the per-library status word by kernels whose waits ran out.
enum StatusCode : int {
  kStatusOk = 0,
  kStatusMbarTimeout = 1,   // an mbarrier wait inside a tcgen05/TMA pipeline gave up
  kStatusPeerTimeout = 2,   // a wait on a flag written by another GPU gave up
  kStatusBadShape = 3,
};

// Number of SMs of the current device (cached per device); grid sizes and per-SM partial buffers derive from it.
inline int device_sm_count() {
  static int sms[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (sms[dev] == 0) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
  return sms[dev] > 0 ? sms[dev] : 148;
}

template <typename T>
struct alignas(16) Vec8 {  // eight 16-bit values = one 128-bit transaction
  T v[8];
};

__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(bf16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ bf16 from_f32<bf16>(float x) { return __float2bfloat16_rn(x); }

// Elements per 128-bit access for a type.
template <typename T> struct VecN { static constexpr int n = 16 / sizeof(T); };

template <typename T, int N>
struct alignas(sizeof(T) * N) Pack {
  T v[N];
};

template <typename T>
__device__ __forceinline__ Pack<T, VecN<T>::n> ld128(const T* p) {
  Pack<T, VecN<T>::n> r;
  *reinterpret_cast<uint4*>(&r) = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <typename T>
__device__ __forceinline__ void st128(T* p, const Pack<T, VecN<T>::n>& r) {
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&r);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  bf162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&t);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  bf162 t = *reinterpret_cast<bf162*>(&u);
  return __bfloat1622float2(t);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum; `red` is shared scratch of >= 32 floats. All threads get the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float r = (lane < nw) ? red[lane] : 0.f;
  r = warp_sum(r);
  return r;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float r = (lane < nw) ? red[lane] : -INFINITY;
  r = warp_max(r);
  return r;
}

// tanh-form GELU used by GPT-2: 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))).
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k = 0.7978845608028654f;
  float u = k * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.f + tanhf(u));
}
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k = 0.7978845608028654f;
  float x2 = x * x;
  float u = k * (x + 0.044715f * x * x2);
  float t = tanhf(u);
  float du = k * (1.f + 3.f * 0.044715f * x2);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}

// two fp32 operations per instruction
__device__ __forceinline__ void fma2(float& a0, float& a1, float b0, float b1, float c0, float c1, float d0, float d1) {
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(a0), "=f"(a1) : "f"(b0), "f"(b1), "f"(c0), "f"(c1), "f"(d0), "f"(d1));
}
__device__ __forceinline__ void mul2(float& a0, float& a1, float b0, float b1, float c0, float c1) {
  asm("{\n\t.reg .b64 x, y;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "mul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(a0), "=f"(a1) : "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void add2(float& a0, float& a1, float b0, float b1, float c0, float c1) {
  asm("{\n\t.reg .b64 x, y;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(a0), "=f"(a1) : "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}

// Programmatic dependent launch.  A kernel that launch_dependent() starts may become resident while the kernel before it in
// the stream still drains: its launch, barrier set-up and tensor memory allocation overlap that tail.  It must call
// dependency_wait() in every thread before the first access to memory that another kernel touches (reads AND writes); the
// wait ends when the kernel before it has completed and its writes are visible, and because that kernel has waited in its
// turn, or was launched in the ordinary way, everything before it has, too.  dependents_launch() allows the next kernel of
// the stream to become resident; it comes after a CTA's own tensor memory allocation, so that the next kernel's CTAs cannot
// get in front of it.  Both do nothing in an ordinary launch.
// Launched this way: kernels with one CTA per SM (GEMM, attention backward), with many waves, or tiny ones.  Not kernels whose
// grid is a few CTAs per SM (column sums, norm backward, element-wise passes): the first SMs to have room would take them
// all (with them, a LLaMA-3 1B step of 4 x 2048 tokens took 77.8 ms instead of 76.3).  Nor kernels that wait for another GPU.
// Measured (B200, captured GPT-2 124M steps): 2 x 128 tokens 3.32 -> 3.06-3.11 ms, 3 x 777 5.20 -> 5.02 ms.
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace titb
