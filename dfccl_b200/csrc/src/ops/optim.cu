// Fused optimizer step over one flat gradient bucket.
//
// The data-parallel engine keeps every bucket as four flat arrays: bf16 (or fp32)
// parameters, their gradients, fp32 master weights and fp32 momentum.  The daemon's
// all-reduce already wrote the averaged gradient in fp32 (scale and cast fused into
// the collective), so the whole update of a bucket is one streaming pass:
//   g = grad + wd * w ; m = mu * m + g ; w -= lr * m ; param = cast(w)
// (SGD with momentum; an AdamW variant of the same shape follows it)
// One launch takes all buckets of a step (a grid of one bucket after the other leaves a ramp up and down of the GPU per
// bucket, and a host call), and clears the buckets' gradients on the way: they sit in arrays of their own that nobody needs
// after the all-reduce, and a fill of its own would be one more launch per bucket.
// Bound: HBM.  22 (SGD) or 30 (AdamW) bytes per element with bf16 parameters, 2 more for the gradient.  What only this kernel
// touches (master weights, moments, the cleared gradients) streams through L2 first to be evicted, so that the reduced gradients the
// all-reduce has just written are still there: ResNet-50's three buckets, all-reduce and SGD, 168.5 -> 165.5 us, with blocks that come up early 163.5.
// No counterpart in the reference, which has no optimizer (it is a collective library); this kernel exists so that the
// gradient path of the benchmarks never leaves flat, heap-resident buffers.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include "dfccl.h"
#include "dfccl_ops.h"
#include "../gemm/tc_common.h"

namespace {

struct OptimArgs {
  dfcclOptimBucket b[DFCCL_OPTIM_MAX_BUCKETS];
  uint32_t firstBlock[DFCCL_OPTIM_MAX_BUCKETS];       // of each bucket
  int n;
  float lr, b1, b2, eps, wd;                           // SGD: b1 is the momentum factor
  float stepSize, invBias2Sqrt;                        // AdamW
  int firstStep;                                       // SGD: the momentum array is not read
};

constexpr int THREADS = 256, UNROLL = 2, PER_BLOCK = THREADS * UNROLL * 4;

// AdamW over the same flat arrays (decoupled weight decay; bias correction folded into the two scalars the host
// passes: stepSize = lr / (1 - beta1^t), invBias2Sqrt = 1 / sqrt(1 - beta2^t)):
//   m = b1 m + (1 - b1) g ; v = b2 v + (1 - b2) g^2 ; w = w (1 - lr wd) - stepSize * m / (sqrt(v) * invBias2Sqrt + eps)
__device__ __forceinline__ void adamwOne(float& w, float g, float& m, float& v, float b1, float b2, float eps, float decay,
                                         float stepSize, float invBias2Sqrt) {
  m = b1 * m + (1.f - b1) * g;
  v = b2 * v + (1.f - b2) * g * g;
  // one square root and one fast division per element: the IEEE division's slow path costs more registers and
  // instructions than the whole rest of the update and made the kernel instruction-bound (2 ulp is irrelevant here)
  w = w * decay - stepSize * __fdividef(m, __fsqrt_rn(v) * invBias2Sqrt + eps);
}

// m <- mu m + (g + wd w), w <- w - lr m
__device__ __forceinline__ void sgdOne(float& w, float g, float& m, float mu, float lr, float wd) {
  g += wd * w;
  m = mu * m + g;
  w -= lr * m;
}

template <bool ADAMW, typename P>
__device__ __forceinline__ void updateBlock(const OptimArgs& a, const dfcclOptimBucket& k, uint32_t block) {
  float* master = (float*)k.master;
  const float* grad = (const float*)k.grad32;
  float* m1 = (float*)k.momentum;
  float* m2 = (float*)k.moment2;
  P* param = (P*)k.param;                                // (fp32 parameters may be the master weights themselves)
  P* clear = (P*)k.clear;
  const float decay = 1.f - a.lr * a.wd;
  const bool fresh = !ADAMW && a.firstStep;
  const size_t nFull = k.n & ~(size_t)3;
  const size_t i0 = (size_t)block * PER_BLOCK + threadIdx.x * 4;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 w[UNROLL], g[UNROLL], m[UNROLL], v[UNROLL];
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    const size_t i = i0 + u * THREADS * 4;
    if (i >= nFull) continue;
    w[u] = __ldcs((const float4*)(master + i));
    g[u] = *(const float4*)(grad + i);
    m[u] = fresh ? zero : __ldcs((const float4*)(m1 + i));
    if (ADAMW) v[u] = __ldcs((const float4*)(m2 + i));
  }
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    const size_t i = i0 + u * THREADS * 4;
    if (i >= nFull) continue;
    if (ADAMW) {
      adamwOne(w[u].x, g[u].x, m[u].x, v[u].x, a.b1, a.b2, a.eps, decay, a.stepSize, a.invBias2Sqrt);
      adamwOne(w[u].y, g[u].y, m[u].y, v[u].y, a.b1, a.b2, a.eps, decay, a.stepSize, a.invBias2Sqrt);
      adamwOne(w[u].z, g[u].z, m[u].z, v[u].z, a.b1, a.b2, a.eps, decay, a.stepSize, a.invBias2Sqrt);
      adamwOne(w[u].w, g[u].w, m[u].w, v[u].w, a.b1, a.b2, a.eps, decay, a.stepSize, a.invBias2Sqrt);
      __stcs((float4*)(m2 + i), v[u]);
    } else {
      sgdOne(w[u].x, g[u].x, m[u].x, a.b1, a.lr, a.wd);
      sgdOne(w[u].y, g[u].y, m[u].y, a.b1, a.lr, a.wd);
      sgdOne(w[u].z, g[u].z, m[u].z, a.b1, a.lr, a.wd);
      sgdOne(w[u].w, g[u].w, m[u].w, a.b1, a.lr, a.wd);
    }
    __stcs((float4*)(master + i), w[u]);
    __stcs((float4*)(m1 + i), m[u]);
    if (sizeof(P) == 2) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(w[u].x, w[u].y), hi = __floats2bfloat162_rn(w[u].z, w[u].w);
      *(uint2*)(param + i) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      if (clear) __stcs((uint2*)(clear + i), make_uint2(0u, 0u));
    } else {
      *(float4*)(param + i) = w[u];
      if (clear) *(float4*)(clear + i) = zero;
    }
  }
  if (block == 0 && threadIdx.x == 0) {                  // up to three elements past the last full pack
    for (size_t i = nFull; i < k.n; ++i) {
      float w1 = master[i], mm = fresh ? 0.f : m1[i];
      if (ADAMW) {
        float vv = m2[i];
        adamwOne(w1, grad[i], mm, vv, a.b1, a.b2, a.eps, decay, a.stepSize, a.invBias2Sqrt);
        m2[i] = vv;
      } else sgdOne(w1, grad[i], mm, a.b1, a.lr, a.wd);
      master[i] = w1; m1[i] = mm;
      if (sizeof(P) == 2) param[i] = (P)__float2bfloat16_rn(w1); else ((float*)param)[i] = w1;
      if (clear) clear[i] = (P)0.f;
    }
  }
}

template <bool ADAMW>
__global__ void __launch_bounds__(THREADS) optimKernel(const __grid_constant__ OptimArgs a) {
  dfccl::tc::grid_dependency_wait();                     // the blocks come up while the kernel in front drains
  dfccl::tc::grid_launch_dependents();
  int j = 0;
  while (j + 1 < a.n && blockIdx.x >= a.firstBlock[j + 1]) ++j;
  const dfcclOptimBucket& k = a.b[j];
  const uint32_t block = blockIdx.x - a.firstBlock[j];
  if (k.paramType == ncclBfloat16) updateBlock<ADAMW, __nv_bfloat16>(a, k, block);
  else updateBlock<ADAMW, float>(a, k, block);
}

// All buckets, as many to a launch as its arguments hold.
template <bool ADAMW>
ncclResult_t run(OptimArgs& a, const dfcclOptimBucket* buckets, int n, cudaStream_t stream) {
  for (int i = 0; i < n; ++i) {
    const dfcclOptimBucket& k = buckets[i];
    if (k.n == 0) continue;
    if (!k.master || !k.grad32 || !k.momentum || !k.param || (ADAMW && !k.moment2)) return ncclInvalidArgument;
    if ((((uintptr_t)k.master | (uintptr_t)k.grad32 | (uintptr_t)k.momentum | (uintptr_t)k.param | (uintptr_t)k.clear | (ADAMW ? (uintptr_t)k.moment2 : 0)) & 15) != 0)
      return ncclInvalidArgument;
    if (k.paramType != ncclBfloat16 && k.paramType != ncclFloat32) return ncclInvalidArgument;
    if ((k.n + PER_BLOCK - 1) / PER_BLOCK > (1u << 30)) return ncclInvalidArgument;
  }
  for (int i = 0; i < n;) {
    uint64_t blocks = 0;
    a.n = 0;
    for (; i < n && a.n < DFCCL_OPTIM_MAX_BUCKETS; ++i) {
      if (buckets[i].n == 0) continue;
      const uint64_t more = (buckets[i].n + PER_BLOCK - 1) / PER_BLOCK;
      if (a.n && blocks + more > (1u << 30)) break;
      a.b[a.n] = buckets[i];
      a.firstBlock[a.n++] = (uint32_t)blocks;
      blocks += more;
    }
    if (!a.n) continue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks); cfg.blockDim = dim3(THREADS); cfg.stream = stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization; at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, optimKernel<ADAMW>, a) != cudaSuccess) { (void)cudaGetLastError(); return ncclUnhandledCudaError; }
  }
  return cudaGetLastError() == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}

}  // namespace

#define DF_API extern "C" __attribute__((visibility("default")))

DF_API ncclResult_t dfcclFusedSgdSteps(const dfcclOptimBucket* buckets, int n, float lr, float mu, float wd, int firstStep, cudaStream_t stream) {
  if (n < 0 || (n > 0 && !buckets)) return ncclInvalidArgument;
  OptimArgs a;
  a.lr = lr; a.b1 = mu; a.wd = wd; a.firstStep = firstStep;
  return run<false>(a, buckets, n, stream);
}

// `step` counts from 1.  State arrays (first and second moment) start at zero.
DF_API ncclResult_t dfcclFusedAdamWSteps(const dfcclOptimBucket* buckets, int n, float lr, float beta1, float beta2, float eps, float wd, int step,
                                         cudaStream_t stream) {
  if (n < 0 || (n > 0 && !buckets) || step < 1) return ncclInvalidArgument;
  OptimArgs a;
  a.lr = lr; a.b1 = beta1; a.b2 = beta2; a.eps = eps; a.wd = wd; a.firstStep = 0;
  a.stepSize = lr / (1.f - powf(beta1, (float)step));
  a.invBias2Sqrt = 1.f / sqrtf(1.f - powf(beta2, (float)step));
  return run<true>(a, buckets, n, stream);
}

// One bucket.  paramType: ncclBfloat16 or ncclFloat32 (then `param` may alias `master`).  All arrays 16-byte aligned.
DF_API ncclResult_t dfcclFusedSgdStep(void* master, const void* grad, void* momentum, void* param, size_t n, int paramType, float lr, float mu, float wd,
                                      int firstStep, cudaStream_t stream) {
  const dfcclOptimBucket b{master, grad, momentum, nullptr, param, nullptr, n, paramType};
  return dfcclFusedSgdSteps(&b, 1, lr, mu, wd, firstStep, stream);
}
DF_API ncclResult_t dfcclFusedAdamWStep(void* master, const void* grad, void* moment1, void* moment2, void* param, size_t n, int paramType, float lr,
                                        float beta1, float beta2, float eps, float wd, int step, cudaStream_t stream) {
  if (n == 0) return ncclSuccess;
  const dfcclOptimBucket b{master, grad, moment1, moment2, param, nullptr, n, paramType};
  return dfcclFusedAdamWSteps(&b, 1, lr, beta1, beta2, eps, wd, step, stream);
}

// Load the kernels of this file into the current context without launching them.
DF_API ncclResult_t dfcclOpsWarm(void) {
  cudaFuncAttributes a;
  if (cudaFuncGetAttributes(&a, optimKernel<false>) != cudaSuccess) return ncclUnhandledCudaError;
  if (cudaFuncGetAttributes(&a, optimKernel<true>) != cudaSuccess) return ncclUnhandledCudaError;
  return ncclSuccess;
}
