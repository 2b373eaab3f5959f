// What a GEMM does with its accumulator before it stores it, for the linear layers of a transformer block.  The persistent
// kernel applies it to the fp32 accumulator; where the product runs on another kernel it is a pass of its own over the
// bf16 result (applyEpilogue).
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace dfccl {

enum GemmEpilogueKind : int {
  EPI_NONE = 0,
  EPI_BIAS = 1,          // C = acc + bias
  EPI_BIAS_RES = 2,      // C = acc + bias + aux                          (aux: the residual, [M, N])
  EPI_BIAS_GELU = 3,     // pre = acc + bias (stored where `pre` is given), C = gelu(pre)     (tanh form)
  EPI_GELU_GRAD = 4,     // C = acc * gelu'(aux)                          (aux: what `pre` was, [M, N])
};
struct GemmEpilogue {
  int kind;
  const __nv_bfloat16* bias;      // [N]
  const __nv_bfloat16* aux;       // [M, N]
  __nv_bfloat16* pre;             // [M, N] or null
};

#if defined(__CUDACC__)
// gelu(x) = x / (1 + exp(-2 z)), z = sqrt(2/pi) (x + 0.044715 x^3): the tanh form without the cancellation of 1 + tanh(z) at
// negative x.  exp and division of the fast kind have errors of a few units in the last place of fp32; the result is
// rounded to bf16.
__device__ __forceinline__ float geluExponent(float x) { return -1.5957691216057308f * (x + 0.044715f * x * x * x); }
__device__ __forceinline__ float geluTanh(float x) { return __fdividef(x, 1.f + __expf(geluExponent(x))); }      // (x / inf = 0 far out)
// d/dx: s + x s (1 - s) 2 z', s = 1 / (1 + e), 1 - s = e s; beyond e^80 it is 0 or 1 in fp32
__device__ __forceinline__ float geluTanhGrad(float x) {
  const float t = geluExponent(x);
  if (t > 80.f) return 0.f;
  if (t < -80.f) return 1.f;
  const float e = __expf(t);
  const float s = __fdividef(1.f, 1.f + e);
  return s + x * s * (e * s) * (1.5957691216057308f + 0.21406453767f * x * x);
}
__device__ __forceinline__ float bf16Lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16Hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
#endif

}  // namespace dfccl
