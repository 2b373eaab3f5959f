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
// gelu(x) = x s, s = 1 / (1 + exp(-2 z)), z = sqrt(2/pi) (x + 0.044715 x^3): the tanh form without the cancellation of
// 1 + tanh(z) at negative x, in seven instructions (the epilogue of a GEMM with a short contraction is bound by them: 8192 x
// 4096 x 1024 took 82 us with __expf and __fdividef).  The two approximations are good to a few units in the last place of
// fp32; the result is rounded to bf16.  Far out the power overflows to infinity and s is 0, or underflows and s is 1.
__device__ __forceinline__ float exp2Approx(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rcpApprox(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// -2 z as a power of two: -2 sqrt(2/pi) log2(e) (x + 0.044715 x^3)
__device__ __forceinline__ float geluPower(float x) { return x * fmaf(x * x, -0.1029432396f, -2.302208198f); }
__device__ __forceinline__ float geluTanh(float x) { return x * rcpApprox(1.f + exp2Approx(geluPower(x))); }
// d/dx: s + x s (1 - s) 2 z', 1 - s = e s; 0 or 1 where e over- or underflows (selected at the end: branches per element cost
// more than the arithmetic)
__device__ __forceinline__ float geluTanhGrad(float x) {
  const float t = geluPower(x), e = exp2Approx(t), s = rcpApprox(1.f + e);
  const float d = fmaf(x * s * (e * s), fmaf(x * x, 0.21406453767f, 1.5957691216057308f), s);
  return t > 115.f ? 0.f : t < -115.f ? 1.f : d;
}
__device__ __forceinline__ float bf16Lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16Hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
#endif

}  // namespace dfccl
