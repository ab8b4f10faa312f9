// Optimizer steps over flat parameter ranges.
//
// Counterpart of infini_train/src/kernels/cuda/accumulate_grad.cu:6-23
// (AccumulateGrad, used for gradient accumulation and as the SGD step) and the
// AdamAccumulateGrad stub at :25-32 whose expected math is the closed form of
// test/optimizer/test_adam.cc:50-58.  One launch covers a whole flat buffer
// (every parameter of a model shard), reads and writes 128 bits per access,
// keeps fp32 master weights and moments, and emits the rounded bf16 copy of the
// weights in the same pass.
#include "api.h"
#include "common.cuh"

namespace titb {

// Bound: memory, 16 bytes read and 14 (bf16 weights) written per parameter.  A CTA updates kAdamPerCta consecutive parameters
// and ends: 4 per thread, the four loads of a thread in flight before the first use, and the five streams of the CTAs that run
// at the same time lie close together (a grid-wide stride spread each stream over the whole buffer).  The state is touched
// once a step and passes through the caches as streaming data; the weights that the next forward pass reads stay.
// Measured (B200, bf16 weights; grid-wide stride -> now): 100 K parameters 2.5 -> 2.2 us, 2 M 7.1 -> 7.1 us, 124 M 631 -> 565 us,
// 780 M 3.97 -> 3.53 ms.  Two vectors per thread and half the CTAs: 2.9 us, 7.5 us, 566 us, 3.54 ms.
constexpr int kAdamVecs = 1;
constexpr int kAdamPerCta = 256 * 4 * kAdamVecs;

template <typename LP>
__global__ void __launch_bounds__(256)
adam_flat_kernel(float* __restrict__ master, LP* __restrict__ lp, const float* __restrict__ grad, float* __restrict__ m,
                 float* __restrict__ v, long long n, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2,
                 float gscale, const float* __restrict__ dev_state) {
  if (dev_state != nullptr) {  // step-dependent scalars kept on the device so a captured graph stays valid
    bc1 = dev_state[1];
    bc2 = dev_state[2];
    lr = dev_state[3];
  }
  const long long base = blockIdx.x * static_cast<long long>(kAdamPerCta) + threadIdx.x * 4;
  float4 g[kAdamVecs], mm[kAdamVecs], vv[kAdamVecs], w[kAdamVecs];
#pragma unroll
  for (int u = 0; u < kAdamVecs; ++u) {
    const long long i = base + u * 1024;
    if (i + 3 < n) {
      g[u] = __ldcs(reinterpret_cast<const float4*>(grad + i));
      mm[u] = __ldcs(reinterpret_cast<const float4*>(m + i));
      vv[u] = __ldcs(reinterpret_cast<const float4*>(v + i));
      w[u] = __ldcs(reinterpret_cast<const float4*>(master + i));
    }
  }
#pragma unroll
  for (int u = 0; u < kAdamVecs; ++u) {
    const long long i = base + u * 1024;
    if (i + 3 < n) {
      float* gp = &g[u].x; float* mp = &mm[u].x; float* vp = &vv[u].x; float* wp = &w[u].x;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float ge = gp[e] * gscale;
        mp[e] = b1 * mp[e] + (1.f - b1) * ge;
        vp[e] = b2 * vp[e] + (1.f - b2) * ge * ge;
        const float mh = mp[e] / bc1, vh = vp[e] / bc2;
        wp[e] -= lr * (mh / (sqrtf(vh) + eps) + wd * wp[e]);
      }
      __stcs(reinterpret_cast<float4*>(m + i), mm[u]);
      __stcs(reinterpret_cast<float4*>(v + i), vv[u]);
      __stcs(reinterpret_cast<float4*>(master + i), w[u]);
      if (lp != nullptr) {
        if constexpr (sizeof(LP) == 2) {
          *reinterpret_cast<uint2*>(lp + i) = make_uint2(pack_bf16x2(wp[0], wp[1]), pack_bf16x2(wp[2], wp[3]));
        } else {
          *reinterpret_cast<float4*>(lp + i) = w[u];
        }
      }
    } else {
      for (long long j = i; j < n; ++j) {
        const float ge = grad[j] * gscale;
        const float mj = b1 * m[j] + (1.f - b1) * ge;
        const float vj = b2 * v[j] + (1.f - b2) * ge * ge;
        m[j] = mj; v[j] = vj;
        const float wj = master[j] - lr * ((mj / bc1) / (sqrtf(vj / bc2) + eps) + wd * master[j]);
        master[j] = wj;
        if (lp != nullptr) lp[j] = from_f32<LP>(wj);
      }
    }
  }
}

// state = {t, 1 - b1^t, 1 - b2^t, lr}; advances t by one.
__global__ void adam_tick_kernel(float* state, float b1, float b2) {
  const float t = state[0] + 1.f;
  state[0] = t;
  state[1] = 1.f - powf(b1, t);
  state[2] = 1.f - powf(b2, t);
}

template <typename LP>
__global__ void sgd_flat_kernel(float* __restrict__ master, LP* __restrict__ lp, const float* __restrict__ grad,
                                long long n, float lr) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float w = master[i] - lr * grad[i];
    master[i] = w;
    if (lp != nullptr) lp[i] = from_f32<LP>(w);
  }
}

template <typename X>
__global__ void axpy_kernel(float* __restrict__ y, const X* __restrict__ x, float a, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] += a * to_f32(x[i]);
}

static inline int blocks_for(long long n) {
  long long b = (n + 255) / 256;
  const long long cap = device_sm_count() * 8;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace titb
using namespace titb;

TITB_API int titb_adam_flat(float* master, void* param_lp, const float* grad, float* m, float* v, long long n, float lr,
                            float beta1, float beta2, float eps, float weight_decay, float bc1, float bc2,
                            float grad_scale, int lp_dtype, const float* dev_state, cudaStream_t st) {
  if (n <= 0) return 0;
  const unsigned blocks = static_cast<unsigned>((n + kAdamPerCta - 1) / kAdamPerCta);
  if (lp_dtype == 1)
    adam_flat_kernel<bf16><<<blocks, 256, 0, st>>>(master, (bf16*)param_lp, grad, m, v, n, lr, beta1, beta2, eps,
                                                   weight_decay, bc1, bc2, grad_scale, dev_state);
  else
    adam_flat_kernel<float><<<blocks, 256, 0, st>>>(master, (float*)param_lp, grad, m, v, n, lr, beta1, beta2, eps,
                                                    weight_decay, bc1, bc2, grad_scale, dev_state);
  return (int)cudaGetLastError();
}

TITB_API int titb_adam_tick(float* state, float beta1, float beta2, cudaStream_t st) {
  adam_tick_kernel<<<1, 1, 0, st>>>(state, beta1, beta2);
  return (int)cudaGetLastError();
}

TITB_API int titb_sgd_flat(float* master, void* param_lp, const float* grad, long long n, float lr, int lp_dtype,
                           cudaStream_t st) {
  if (n <= 0) return 0;
  if (lp_dtype == 1) sgd_flat_kernel<bf16><<<blocks_for(n), 256, 0, st>>>(master, (bf16*)param_lp, grad, n, lr);
  else sgd_flat_kernel<float><<<blocks_for(n), 256, 0, st>>>(master, (float*)param_lp, grad, n, lr);
  return (int)cudaGetLastError();
}

TITB_API int titb_axpy(float* y, const void* x, float a, long long n, int x_dtype, cudaStream_t st) {
  if (n <= 0) return 0;
  if (x_dtype == 1) axpy_kernel<bf16><<<blocks_for(n), 256, 0, st>>>(y, (const bf16*)x, a, n);
  else axpy_kernel<float><<<blocks_for(n), 256, 0, st>>>(y, (const float*)x, a, n);
  return (int)cudaGetLastError();
}
