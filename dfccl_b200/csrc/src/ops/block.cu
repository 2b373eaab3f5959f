// Elementwise and row / column work of a transformer block around its GEMMs, bf16 in and out, fp32 inside: layer norm
// forward and backward, column sums (bias gradients), and the GEMM epilogues as passes of their own.
// All of it streams activations once, so HBM (or L2) bounds it: 16 bytes per load, every row in registers between its two
// passes, and enough warps to keep 148 SMs loading.  The measured times stand at the kernels.
// They are short and follow one another: each (but the epilogue pass) is launched as a dependent of the kernel in front, so that its
// blocks are up when that one ends.
// The reference has no counterpart (it is a collective library); the GPT-2 workload uses these.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include "dfccl.h"
#include "../common/device_once.h"
#include "../gemm/epilogue.h"
#include "../gemm/gemm.h"
#include "../gemm/tc_common.h"

namespace dfccl {
namespace {

constexpr int MAX_D = 2048;            // widest row a warp keeps in registers (8 packs of 8 elements per lane)

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& p, float (&f)[8]) {
  const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { f[2 * i] = bf16Lo(w[i]); f[2 * i + 1] = bf16Hi(w[i]); }
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}

// One warp per row; NV packs of 8 elements per lane (d <= 256 NV, a multiple of 8).
template <int NV>
__global__ void __launch_bounds__(128) lnForwardKernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                                                       const __nv_bfloat16* __restrict__ beta, __nv_bfloat16* __restrict__ y,
                                                       float* __restrict__ mean, float* __restrict__ rstd, int rows, int d, float eps) {
  const int lane = threadIdx.x & 31, row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  tc::grid_dependency_wait();
  tc::grid_launch_dependents();
  const uint4* src = (const uint4*)(x + (size_t)row * d);
  uint4 p[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) { const int i = v * 32 + lane; p[v] = i * 8 < d ? src[i] : make_uint4(0u, 0u, 0u, 0u); }
  float s = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    float f[8];
    unpack8(p[v], f);
#pragma unroll
    for (int e = 0; e < 8; ++e) s += f[e];
  }
  const float m = warpSum(s) / d;
  float q = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    if ((v * 32 + lane) * 8 >= d) continue;
    float f[8];
    unpack8(p[v], f);
#pragma unroll
    for (int e = 0; e < 8; ++e) q += (f[e] - m) * (f[e] - m);
  }
  const float r = rsqrtf(warpSum(q) / d + eps);
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int i = v * 32 + lane;
    if (i * 8 >= d) continue;
    float f[8], g[8], b[8], o[8];
    unpack8(p[v], f); unpack8(__ldg((const uint4*)gamma + i), g); unpack8(__ldg((const uint4*)beta + i), b);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = (f[e] - m) * r * g[e] + b[e];
    ((uint4*)(y + (size_t)row * d))[i] = pack8(o);
  }
  if (lane == 0) { mean[row] = m; rstd[row] = r; }
}

// 8192 x 1024 (16.8 MB a tensor, four of them here), us: 15.8 with the line sums; row by row without loads ahead, the warps
// adding up in turns, it was 36, the two framework kernels it replaces 57 and their residual add 7.  Forward: 6.3 (22.5).
// gx = rstd (gy gamma - mean(gy gamma) - xhat mean(gy gamma xhat)) [+ pass].  A warp takes every (8 x blocks)-th row with the
// next row's loads in flight, and keeps its rows' sums of gy xhat and gy in registers; a block adds its warps' through shared
// memory and writes one line of `work`, [blocks][2][d].
template <int NV>
__global__ void __launch_bounds__(256, 1) lnBackwardKernel(const __nv_bfloat16* __restrict__ gy, const __nv_bfloat16* __restrict__ x,
                                                           const __nv_bfloat16* __restrict__ gamma, const float* __restrict__ mean,
                                                           const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ pass,
                                                           __nv_bfloat16* __restrict__ gx, float* __restrict__ work, int rows, int d) {
  constexpr bool AHEAD = NV <= 4;                        // (the widest rows would not leave the registers for it)
  extern __shared__ float sums[];                        // [8 warps][2][d]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, step = gridDim.x * 8;
  tc::grid_dependency_wait();
  tc::grid_launch_dependents();
  float dg[NV][8], db[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int e = 0; e < 8; ++e) { dg[v][e] = 0.f; db[v][e] = 0.f; }
  uint4 pg[NV], px[NV], pp[NV];
  float m, r;
  auto load = [&](int row) {
    const size_t off = (size_t)row * d;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int i = v * 32 + lane;
      const bool in = i * 8 < d;
      pg[v] = in ? ((const uint4*)(gy + off))[i] : make_uint4(0u, 0u, 0u, 0u);
      px[v] = in ? ((const uint4*)(x + off))[i] : make_uint4(0u, 0u, 0u, 0u);
      pp[v] = in && pass ? ((const uint4*)(pass + off))[i] : make_uint4(0u, 0u, 0u, 0u);
    }
    m = mean[row]; r = rstd[row];
  };
  int row = blockIdx.x * 8 + warp;
  if (AHEAD && row < rows) load(row);
  for (; row < rows; row += step) {
    if (!AHEAD) load(row);
    uint4 cg[NV], cx[NV], cp[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) { cg[v] = pg[v]; cx[v] = px[v]; cp[v] = pp[v]; }
    const float cm = m, crs = r;
    if (AHEAD && row + step < rows) load(row + step);
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int i = v * 32 + lane;
      if (i * 8 >= d) continue;
      float g[8], f[8], w[8];
      unpack8(cg[v], g); unpack8(cx[v], f); unpack8(__ldg((const uint4*)gamma + i), w);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float xh = (f[e] - cm) * crs, gw = g[e] * w[e];
        s1 += gw; s2 += gw * xh;
        dg[v][e] += g[e] * xh; db[v][e] += g[e];
      }
    }
    s1 = warpSum(s1) / d; s2 = warpSum(s2) / d;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int i = v * 32 + lane;
      if (i * 8 >= d) continue;
      float g[8], f[8], w[8], p[8], o[8];
      unpack8(cg[v], g); unpack8(cx[v], f); unpack8(__ldg((const uint4*)gamma + i), w); unpack8(cp[v], p);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = crs * (g[e] * w[e] - s1 - (f[e] - cm) * crs * s2) + p[e];
      ((uint4*)(gx + (size_t)row * d))[i] = pack8(o);
    }
  }
  float* mine = sums + warp * 2 * d;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int i = (v * 32 + lane) * 8;
    if (i >= d) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      *(float4*)(mine + i + 4 * h) = make_float4(dg[v][4 * h], dg[v][4 * h + 1], dg[v][4 * h + 2], dg[v][4 * h + 3]);
      *(float4*)(mine + d + i + 4 * h) = make_float4(db[v][4 * h], db[v][4 * h + 1], db[v][4 * h + 2], db[v][4 * h + 3]);
    }
  }
  __syncthreads();
  float* line = work + (size_t)blockIdx.x * 2 * d;
  for (int i = threadIdx.x; i < 2 * d; i += 256) {
    float s = sums[i];
#pragma unroll
    for (int w = 1; w < 8; ++w) s += sums[w * 2 * d + i];
    line[i] = s;
  }
}

// out[c] = sum over lines of work[line][c], 32 columns per block, 32 lines at a time; columns from `split` on go to out2.
__global__ void __launch_bounds__(1024) sumLinesKernel(const float* __restrict__ work, int lines, int n, __nv_bfloat16* __restrict__ out,
                                                       __nv_bfloat16* __restrict__ out2, int split) {
  __shared__ float part[32][33];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  tc::grid_dependency_wait();
  tc::grid_launch_dependents();
  if (c < n) {
#pragma unroll 4
    for (int l = g; l < lines; l += 32) s += work[(size_t)l * n + c];
  }
  part[g][lane] = s;
  __syncthreads();
  s = warpSum(part[lane][g]);                            // warp g adds column g of the block's 32
  const int col = blockIdx.x * 32 + g;
  if (lane == 0 && col < n) {
    if (col < split) out[col] = __float2bfloat16_rn(s); else out2[col - split] = __float2bfloat16_rn(s);
  }
}

// Sums of 64 columns from c0 on over rows [beg, end) by a block of 256 threads, in `sums`: a warp reads four rows of 128 bytes at a
// time, eight such loads in flight, the block adds its warps up through shared memory in a fixed order.
struct ColumnShared { float part[8][4][64 + 4], sums[64]; };
__device__ __forceinline__ void sumColumns(ColumnShared& sh, const __nv_bfloat16* __restrict__ g, int beg, int end, int n, int c0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = c0 + (lane & 7) * 8;
  float a[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) a[e] = 0.f;
  if (c < n) {
#pragma unroll 8
    for (int r = beg + warp * 4 + (lane >> 3); r < end; r += 32) {
      float f[8];
      unpack8(*(const uint4*)(g + (size_t)r * n + c), f);
#pragma unroll
      for (int e = 0; e < 8; ++e) a[e] += f[e];
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) sh.part[warp][lane >> 3][(lane & 7) * 8 + e] = a[e];
  __syncthreads();
  if (threadIdx.x < 64) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w)
#pragma unroll
      for (int q = 0; q < 4; ++q) s += sh.part[w][q][threadIdx.x];
    sh.sums[threadIdx.x] = s;
  }
  __syncthreads();
}

// Column sums in one launch: a cluster of SUM_CTAS blocks takes 64 columns, a stretch of the rows each, and the cluster's blocks
// write 64 / SUM_CTAS columns each from one another's shared memory.  No scratch in global memory, no second kernel, a
// fixed order of the sums.  Bound: one read of the matrix.  us behind a kernel that rewrites it, two launches with scratch memory
// / this: 8192 x 1024 5.9 / 4.8, 8192 x 3072 8.0 / 6.4, 8192 x 4096 9.4 / 7.9.
constexpr int SUM_CTAS = 8;
__global__ void __cluster_dims__(SUM_CTAS, 1, 1) __launch_bounds__(256) columnSumKernel(const __nv_bfloat16* __restrict__ g, __nv_bfloat16* __restrict__ out, int rows, int n) {
  __shared__ ColumnShared sh;
  const int rank = blockIdx.x % SUM_CTAS, c0 = blockIdx.x / SUM_CTAS * 64;
  const int per = (rows + SUM_CTAS - 1) / SUM_CTAS, beg = rank * per, end = min(rows, beg + per);
  tc::grid_dependency_wait();
  tc::grid_launch_dependents();
  sumColumns(sh, g, beg, end, n, c0);
  tc::cluster_sync_all();                                // every block's sums are there
  if (threadIdx.x < 64 / SUM_CTAS) {
    const int k = rank * (64 / SUM_CTAS) + threadIdx.x;
    float s = 0.f;
#pragma unroll
    for (int b = 0; b < SUM_CTAS; ++b) {
      float v;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(tc::mapa_u32(tc::smem_u32(&sh.sums[k]), b)) : "memory");
      s += v;
    }
    if (c0 + k < n) out[c0 + k] = __float2bfloat16_rn(s);
  }
  tc::cluster_sync_all();                                // nobody reads this block's shared memory any more
}

// The same for matrices too narrow for their height (sumStretches): gridDim.y stretches of rows, a line of fp32 sums in `work`
// each, which sumLinesKernel adds up.
__global__ void __launch_bounds__(256) columnLinesKernel(const __nv_bfloat16* __restrict__ g, float* __restrict__ work, int rows, int n) {
  __shared__ ColumnShared sh;
  const int per = (rows + gridDim.y - 1) / gridDim.y, beg = blockIdx.y * per, end = min(rows, beg + per), c = blockIdx.x * 64 + threadIdx.x;
  tc::grid_dependency_wait();
  tc::grid_launch_dependents();
  sumColumns(sh, g, beg, end, n, blockIdx.x * 64);
  if (threadIdx.x < 64 && c < n) work[(size_t)blockIdx.y * n + c] = sh.sums[threadIdx.x];
}

template <int EPI>
__global__ void __launch_bounds__(256) epilogueKernel(GemmEpilogue e, __nv_bfloat16* __restrict__ C, size_t packs, int packsPerRow) {
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < packs; i += (size_t)gridDim.x * 256) {
    float v[8], b[8], x[8];
    unpack8(((const uint4*)C)[i], v);
    if (EPI == EPI_BIAS || EPI == EPI_BIAS_RES || EPI == EPI_BIAS_GELU) {
      unpack8(__ldg((const uint4*)e.bias + i % packsPerRow), b);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += b[k];
    }
    if (EPI == EPI_BIAS_RES || EPI == EPI_GELU_GRAD) {
      unpack8(((const uint4*)e.aux)[i], x);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = EPI == EPI_BIAS_RES ? v[k] + x[k] : v[k] * geluTanhGrad(x[k]);
    }
    if (EPI == EPI_BIAS_GELU) {
      const uint4 p = pack8(v);
      if (e.pre) ((uint4*)e.pre)[i] = p;
      unpack8(p, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = geluTanh(v[k]);
    }
    ((uint4*)C)[i] = pack8(v);
  }
}

int smCount() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}
ncclResult_t launched() { return cudaGetLastError() == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError; }
bool aligned(const void* a, const void* b = nullptr, const void* c = nullptr, const void* d = nullptr, const void* e = nullptr) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d | (uintptr_t)e) & 15) == 0;
}
int lnBlocks(int rows, int sms) { return std::max(1, std::min((rows + 7) / 8, sms)); }
// Stretches of rows of a column sum; 0: one launch of clusters.  A block of a cluster sums an eighth of the rows however many there
// are, and a narrow matrix has few clusters: from 16384 rows on and up to 1984 columns (fewer than 256 blocks of clusters) the rows
// are cut into what gives every SM two blocks.  us behind a kernel that rewrites the matrix, clusters / stretches: 8192 x 1024 4.8 / 5.8,
// 16384 x 256 6.7 / 5.7, 16384 x 1024 7.8 / 7.0, 16384 x 1536 8.0 / 7.8, 65536 x 256 18.6 / 6.7, 32768 x 768 11.0 / 7.7, 65536 x 1536
// 41.4 / 34.9, 16384 x 2048 8.8 / 8.7, 24576 x 2048 15.9 / 16.7, 16384 x 3072 13.4 / 17.0; four or eight blocks an SM are slower.
int sumStretches(int rows, int n, int sms) {
  const int groups = (n + 63) / 64;
  if (rows < 16384 || groups * SUM_CTAS >= 256) return 0;
  return std::max(1, std::min(2 * sms / groups, rows / 128));
}
// Launched so that the blocks may come up while the kernel in front still drains (tc_common.h: grid_dependency_wait).
template <typename... P, typename... A>
cudaError_t launchBehind(void (*kernel)(P...), dim3 grid, int block, int smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization; at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

template <int NV>
cudaError_t lnBackward(const void* gy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* pass, void* gx, float* work,
                int rows, int d, int blocks, cudaStream_t stream) {
  const int smem = 8 * 2 * d * (int)sizeof(float);
  // (up to 128 KB for the widest rows)
  const cudaError_t e = oncePerDevice([] { return allowSharedMemory(lnBackwardKernel<NV>, 8 * 2 * 256 * NV * (int)sizeof(float)); });
  if (e != cudaSuccess) return e;
  return launchBehind(lnBackwardKernel<NV>, blocks, 256, smem, stream, (const __nv_bfloat16*)gy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)gamma,
                      mean, rstd, (const __nv_bfloat16*)pass, (__nv_bfloat16*)gx, work, rows, d);
}

}  // namespace

ncclResult_t applyEpilogue(const GemmEpilogue& e, void* C, int M, int N, cudaStream_t stream) {
  const size_t packs = (size_t)M * N / 8;
  const unsigned grid = (unsigned)std::min<size_t>((packs + 255) / 256, (size_t)smCount() * 8);
  switch (e.kind) {
    case EPI_BIAS: epilogueKernel<EPI_BIAS><<<grid, 256, 0, stream>>>(e, (__nv_bfloat16*)C, packs, N / 8); break;
    case EPI_BIAS_RES: epilogueKernel<EPI_BIAS_RES><<<grid, 256, 0, stream>>>(e, (__nv_bfloat16*)C, packs, N / 8); break;
    case EPI_BIAS_GELU: epilogueKernel<EPI_BIAS_GELU><<<grid, 256, 0, stream>>>(e, (__nv_bfloat16*)C, packs, N / 8); break;
    case EPI_GELU_GRAD: epilogueKernel<EPI_GELU_GRAD><<<grid, 256, 0, stream>>>(e, (__nv_bfloat16*)C, packs, N / 8); break;
    default: return ncclSuccess;
  }
  return launched();
}

}  // namespace dfccl

using namespace dfccl;
#define DF_API extern "C" __attribute__((visibility("default")))

// Widest row of the layer norm kernels (a multiple of 8 elements).
DF_API int dfcclLayerNormMaxWidth(void) { return MAX_D; }

// y = (x - mean) rstd gamma + beta per row of d elements; mean and rstd [rows] fp32 for the backward pass.
DF_API ncclResult_t dfcclLayerNormForward(const void* x, const void* gamma, const void* beta, void* y, void* mean, void* rstd, int rows, int d, float eps, cudaStream_t stream) {
  if (rows <= 0 || d <= 0 || d % 8 || d > MAX_D || !x || !gamma || !beta || !y || !mean || !rstd || !aligned(x, gamma, beta, y)) return ncclInvalidArgument;
  auto* kernel = d <= 256 ? lnForwardKernel<1> : d <= 512 ? lnForwardKernel<2> : d <= 1024 ? lnForwardKernel<4> : lnForwardKernel<8>;
  const cudaError_t e = launchBehind(kernel, (rows + 3) / 4, 128, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)gamma, (const __nv_bfloat16*)beta,
                                     (__nv_bfloat16*)y, (float*)mean, (float*)rstd, rows, d, eps);
  return e == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}

// fp32 words of scratch memory a backward pass / a column sum needs on the current device.
DF_API size_t dfcclLayerNormWork(int rows, int d) { return (size_t)lnBlocks(rows, smCount()) * 2 * d; }
DF_API size_t dfcclColumnSumWork(int rows, int n) { return rows <= 0 || n <= 0 ? 0 : (size_t)sumStretches(rows, n, smCount()) * n; }

// Gradients of x (plus `pass`, the gradient that reaches x by another way, where given), gamma and beta.
DF_API ncclResult_t dfcclLayerNormBackward(const void* gy, const void* x, const void* gamma, const void* mean, const void* rstd, const void* pass,
                                           void* gx, void* ggamma, void* gbeta, void* work, int rows, int d, cudaStream_t stream) {
  if (rows <= 0 || d <= 0 || d % 8 || d > MAX_D || !gy || !x || !gamma || !mean || !rstd || !gx || !ggamma || !gbeta || !work) return ncclInvalidArgument;
  if (!aligned(gy, x, gamma, pass, gx)) return ncclInvalidArgument;
  const int blocks = lnBlocks(rows, smCount());
  auto* fn = d <= 256 ? lnBackward<1> : d <= 512 ? lnBackward<2> : d <= 1024 ? lnBackward<4> : lnBackward<8>;
  if (fn(gy, x, gamma, (const float*)mean, (const float*)rstd, pass, gx, (float*)work, rows, d, blocks, stream) != cudaSuccess) return ncclUnhandledCudaError;
  const cudaError_t e = launchBehind(sumLinesKernel, (2 * d + 31) / 32, 1024, 0, stream, (const float*)work, blocks, 2 * d, (__nv_bfloat16*)ggamma, (__nv_bfloat16*)gbeta, d);
  return e == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}

// out[n] = sum over rows of g [rows, n], added up in fp32.  `work`: dfcclColumnSumWork words (null: in one launch whatever the shape).
DF_API ncclResult_t dfcclColumnSum(const void* g, void* out, void* work, int rows, int n, cudaStream_t stream) {
  if (rows <= 0 || n <= 0 || n % 8 || !g || !out || !aligned(g)) return ncclInvalidArgument;
  const int groups = (n + 63) / 64, stretches = work ? sumStretches(rows, n, smCount()) : 0;
  cudaError_t e;
  if (stretches) {
    e = launchBehind(columnLinesKernel, dim3(groups, stretches), 256, 0, stream, (const __nv_bfloat16*)g, (float*)work, rows, n);
    if (e == cudaSuccess) e = launchBehind(sumLinesKernel, (n + 31) / 32, 1024, 0, stream, (const float*)work, stretches, n, (__nv_bfloat16*)out, (__nv_bfloat16*)out, n);
  } else {
    e = launchBehind(columnSumKernel, groups * SUM_CTAS, 256, 0, stream, (const __nv_bfloat16*)g, (__nv_bfloat16*)out, rows, n);
  }
  return e == cudaSuccess ? ncclSuccess : ncclUnhandledCudaError;
}
