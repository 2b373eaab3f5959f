// bf16 GEMM on CTA pairs (tcgen05 cta_group::2), hand-written for sm_100a:
//     C[M,N] = A[M,K] * B[N,K]^T,  tiles of 256 x 256, one tile per pair of CTAs (a cluster of two SMs).  Rows of the last
//     row tile beyond M (M is a multiple of 128) are loaded as zeros and not stored.
// Each CTA of a pair loads 128 rows of A and 128 rows of B per 64-wide K block (32 KB per stage instead of the 48 KB
// of the one-CTA form, so six stages fit), the leader's single MMA thread issues 256 x 256 x 16 instructions that read
// both CTAs' shared memory, and each CTA ends up with its 128 rows of the accumulator in its own tensor memory.
// The tensor cores of an SM thus see every B row once per pair instead of once per CTA: half the shared-memory
// operand traffic per FLOP, which is what bounds the one-CTA kernel.
//
// Roles per CTA: warp 0 = TMA producer (one elected thread; completion of both CTAs' loads is counted on the
// LEADER's barrier), warp 1 = tensor-memory owner, and in the leader the MMA issuer; warps 2-9 = epilogue over the
// CTA's own accumulator half.  Stages are released and accumulators handed over with tcgen05.commit to both CTAs;
// the epilogues of both CTAs arrive on the leader's accumulator-empty barrier.  No TMA load uses cluster multicast.
// Every wait is bounded and ends in the error word of the device.
//
// The reference has no tensor-core code (it is a collective library); this kernel serves the tensor-parallel
// workloads' plain GEMMs (weight and data gradients, unfused forwards).
#include "tc_common.h"
#include "gemm.h"
#include "epilogue.h"
#include "../common/device_once.h"
#include "../common/param.h"
#include "../common/log.h"
#include <algorithm>
#include <mutex>

namespace dfccl {
namespace {

using namespace tc;

constexpr int PM = 256, PN = 256, BK = 64, HALF = 128, STAGES = 6, UMMA_K = 16;
constexpr int A_BYTES = HALF * BK * 2, B_BYTES = HALF * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;   // per CTA
constexpr int MN_BLOCK_BYTES = 64 * BK * 2;
constexpr int TMEM_COLS = 512;                       // two accumulators of 256 fp32 columns (128 lanes each, per CTA)
constexpr int NUM_THREADS = 320;                     // 10 warps
constexpr int EPI_WARPS = 8;                         // two per 32 accumulator rows: the last tile's epilogue is not overlapped with anything
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr uint64_t WAIT_NS = 4000000000ull;          // nothing here waits on another GPU: seconds mean a lost partner

struct PairArgs {
  __nv_bfloat16* C;
  int M, N, K, ldc;
  int aMn, bMn;
  int groupM;                       // row tiles per rasterisation group
  uint32_t* err;
  uint32_t* errHost;
  GemmEpilogue e;
  bool wide;                        // C, aux and pre start on 32-byte boundaries
};

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
dfcclGemmPairKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const PairArgs g) {
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint64_t* fullBar = (uint64_t*)(smem + STAGES * STAGE_BYTES);     // used in the leader only
  uint64_t* emptyBar = fullBar + STAGES;                             // in both CTAs (commit to both)
  uint64_t* accFull = emptyBar + STAGES;                             // [2] in both CTAs
  uint64_t* accEmpty = accFull + 2;                                  // [2] used in the leader only: the epilogue warps of both CTAs arrive
  uint32_t* tmemBaseSlot = (uint32_t*)(accEmpty + 2);
  volatile uint32_t* giveUp = tmemBaseSlot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cr = cluster_ctarank();             // 0 = leader
  const int mTiles = (g.M + PM - 1) / PM, nTiles = g.N / PN, kBlocks = g.K / BK;
  const int numTiles = mTiles * nTiles;
  const int pair = blockIdx.x >> 1, numPairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&fullBar[s], 1); mbar_init(&emptyBar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&accFull[a], 1); mbar_init(&accEmpty[a], 2 * EPI_WARPS); }
    // (not the device's error word: read here, beside the kernel in front, it could differ between the two CTAs, and one would
    // wait for a partner that does nothing.  After a kernel has given up the host refuses launches.)
    *giveUp = 0;
    mbar_fence_init();
    tma_prefetch_desc(&mapA);
    tma_prefetch_desc(&mapB);
  }
  if (warp == 1) tmem_alloc_pair(tmemBaseSlot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                // the partner's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmemBase = *tmemBaseSlot;
  grid_dependency_wait();                            // everything above may run beside the kernel in front of this one
  grid_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs; bytes counted in the leader)
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += numPairs) {
        int mt, nt;
        raster_tile(t, mTiles, nTiles, g.groupM, mt, nt);
        const int rowA = mt * PM + (int)cr * HALF, rowB = nt * PN + (int)cr * HALF;
        for (int kb = 0; kb < kBlocks; ++kb) {
          if (!mbar_wait(&emptyBar[stage], phase ^ 1, giveUp, WAIT_NS)) { ok = false; break; }
          if (cr == 0) mbar_expect_tx(&fullBar[stage], 2 * STAGE_BYTES);        // my bytes and the partner's
          const uint32_t bar = mapa_u32(smem_u32(&fullBar[stage]), 0);
          uint8_t* sa = smem + stage * STAGE_BYTES;
          if (!g.aMn) tma_load_2d_pair(sa, &mapA, kb * BK, rowA, bar);
          else for (int i = 0; i < HALF / 64; ++i) tma_load_2d_pair(sa + i * MN_BLOCK_BYTES, &mapA, rowA + 64 * i, kb * BK, bar);
          if (!g.bMn) tma_load_2d_pair(sa + A_BYTES, &mapB, kb * BK, rowB, bar);
          else for (int i = 0; i < HALF / 64; ++i) tma_load_2d_pair(sa + A_BYTES + i * MN_BLOCK_BYTES, &mapB, rowB + 64 * i, kb * BK, bar);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) for (int i = 0; i < 20000; ++i) __nanosleep(200);     // copies already issued land before the CTA goes away
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (cr == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(PM, PN, g.aMn, g.bMn);
      const uint32_t stepA = g.aMn ? 128u : 2u, stepB = g.bMn ? 128u : 2u;
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += numPairs, ++it) {
        const int ab = it & 1;
        if (!mbar_wait(&accEmpty[ab], ((it >> 1) & 1) ^ 1, giveUp, WAIT_NS)) break;
        tc_fence_after();
        const uint32_t d = tmemBase + ab * PN;
        for (int kb = 0; kb < kBlocks; ++kb) {
          if (!mbar_wait(&fullBar[stage], phase, giveUp, WAIT_NS)) { ok = false; break; }
          tc_fence_after();
          const uint8_t* pa = smem + stage * STAGE_BYTES;
          const uint64_t da = g.aMn ? umma_smem_desc_mn_sw128(pa, MN_BLOCK_BYTES) : umma_smem_desc_sw128(pa);
          const uint64_t db = g.bMn ? umma_smem_desc_mn_sw128(pa + A_BYTES, MN_BLOCK_BYTES) : umma_smem_desc_sw128(pa + A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_pair(d, da + stepA * k, db + stepB * k, idesc, (kb | k) != 0);
          umma_commit_pair(&emptyBar[stage]);         // both CTAs' stage is free once these MMAs have read it
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit_pair(&accFull[ab]);       // both halves of the accumulator complete
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: my 128 rows, TMEM -> bf16 -> global
    const int quarter = warp & 3, colHalf = (warp - 2) >> 2;
    const uint32_t accEmptyLeader0 = mapa_u32(smem_u32(&accEmpty[0]), 0), accEmptyLeader1 = mapa_u32(smem_u32(&accEmpty[1]), 0);
    int it = 0;
    for (int t = pair; t < numTiles; t += numPairs, ++it) {
      int mt, nt;
      raster_tile(t, mTiles, nTiles, g.groupM, mt, nt);
      const int ab = it & 1;
      const bool mine = mt * PM + (int)cr * HALF < g.M;               // the last row tile may have only its upper half
      const size_t tileOff = (size_t)(mt * PM + (int)cr * HALF + quarter * 32) * g.ldc + nt * PN;   // row 0 of this warp's 32 rows
      const int beg = colHalf * (PN / 2);
      // 32 columns of its row per lane and step, 32 bytes (a whole sector) per access: no staging rows, whose way through
      // shared memory the operands need (8192 x 4096 x 1024 with GELU's gradient: 105 -> 70 - 79 us, by run)
      constexpr bool AUX = EPI == EPI_BIAS_RES || EPI == EPI_GELU_GRAD;
      constexpr int STEPS = PN / 2 / 32;
      const size_t mineOff = tileOff + (size_t)lane * g.ldc + beg;
      if (!mbar_wait(&accFull[ab], (it >> 1) & 1, giveUp, WAIT_NS)) break;
      tc_fence_after();
#pragma unroll 1
      for (int i = 0; i < STEPS; ++i) {
        if (!mine) break;
        const int c = beg + i * 32;
        uint32_t r[32];
        tmem_ld32(tmemBase + ((uint32_t)(quarter * 32) << 16) + ab * PN + c, r);
        uint4 own[4];
        if (AUX) {
          ld_global32(g.e.aux + mineOff + i * 32, own, g.wide);
          ld_global32(g.e.aux + mineOff + i * 32 + 16, own + 2, g.wide);
        }
        tmem_ld_wait();
        if (EPI == EPI_BIAS || EPI == EPI_BIAS_RES || EPI == EPI_BIAS_GELU) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const uint4 bv = ((const uint4*)(g.e.bias + nt * PN + c))[v];
            const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              r[8 * v + 2 * w] = __float_as_uint(__uint_as_float(r[8 * v + 2 * w]) + bf16Lo(bw[w]));
              r[8 * v + 2 * w + 1] = __float_as_uint(__uint_as_float(r[8 * v + 2 * w + 1]) + bf16Hi(bw[w]));
            }
          }
        }
        if (AUX) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const uint32_t xw[4] = {own[v].x, own[v].y, own[v].z, own[v].w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              float lo = __uint_as_float(r[8 * v + 2 * w]), hi = __uint_as_float(r[8 * v + 2 * w + 1]);
              if (EPI == EPI_BIAS_RES) { lo += bf16Lo(xw[w]); hi += bf16Hi(xw[w]); }
              else { lo *= geluTanhGrad(bf16Lo(xw[w])); hi *= geluTanhGrad(bf16Hi(xw[w])); }
              r[8 * v + 2 * w] = __float_as_uint(lo); r[8 * v + 2 * w + 1] = __float_as_uint(hi);
            }
          }
        }
        uint4 o[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          o[v].x = pack_bf16x2(__uint_as_float(r[8 * v + 0]), __uint_as_float(r[8 * v + 1]));
          o[v].y = pack_bf16x2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3]));
          o[v].z = pack_bf16x2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5]));
          o[v].w = pack_bf16x2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7]));
        }
        if (EPI == EPI_BIAS_GELU) {
          if (g.e.pre) {
            st_global32(g.e.pre + mineOff + i * 32, o, g.wide);
            st_global32(g.e.pre + mineOff + i * 32 + 16, o + 2, g.wide);
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {                // of the rounded value: what the backward pass differentiates at
            uint32_t* ow = (uint32_t*)&o[v];
#pragma unroll
            for (int w = 0; w < 4; ++w) ow[w] = pack_bf16x2(geluTanh(bf16Lo(ow[w])), geluTanh(bf16Hi(ow[w])));
          }
        }
        st_global32(g.C + mineOff + i * 32, o, g.wide);
        st_global32(g.C + mineOff + i * 32 + 16, o + 2, g.wide);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(ab ? accEmptyLeader1 : accEmptyLeader0);   // the pair's epilogue warps release the accumulator
    }
  }

  // ---------------------------------------------------------------- leave: nothing of the pair may still use my shared or tensor memory
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmemBase, TMEM_COLS);
  if (threadIdx.x == 0 && *giveUp) { atomicExch(g.err, 1u); *(volatile uint32_t*)g.errHost = 1u; __threadfence_system(); }
}

}  // namespace

namespace {
typedef void (*PairKernel)(const CUtensorMap, const CUtensorMap, const PairArgs);
PairKernel pairKernel(int epi) {
  static const PairKernel k[] = {dfcclGemmPairKernel<EPI_NONE>, dfcclGemmPairKernel<EPI_BIAS>, dfcclGemmPairKernel<EPI_BIAS_RES>,
                                 dfcclGemmPairKernel<EPI_BIAS_GELU>, dfcclGemmPairKernel<EPI_GELU_GRAD>};
  return k[epi];
}
cudaError_t allowPairs() {
  return oncePerDevice([] {
    cudaError_t r = cudaSuccess;
    for (int e = EPI_NONE; e <= EPI_GELU_GRAD && r == cudaSuccess; ++e) r = allowSharedMemory(pairKernel(e), SMEM_BYTES);
    return r;
  });
}
int maxResidentPairs(int dev, int sms) {
  // pairs that can be resident together (a GPC with an odd number of free SMs leaves one unpaired)
  static int maxPairs[64];
  static std::mutex mu;
  std::lock_guard<std::mutex> l(mu);
  if (!maxPairs[dev & 63]) {
    (void)allowPairs();                                // (the launch reports it)
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(sms & ~1); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = SMEM_BYTES;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, pairKernel(EPI_NONE), &cfg) != cudaSuccess || n <= 0) { (void)cudaGetLastError(); n = sms / 2; }
    maxPairs[dev & 63] = std::min(n, sms / 2);
  }
  return maxPairs[dev & 63];
}
}  // namespace

int gemmPairResident() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return maxResidentPairs(dev, sms);
}

ncclResult_t gemmPairLaunch(const void* A, const void* B, void* C, int M, int N, int K, cudaStream_t stream, int aMn, int bMn,
                            uint32_t* errDev, uint32_t* errHost, const GemmEpilogue* e) {
  CUtensorMap ma, mb;
  if (!aMn) DFCHECK(gemmMakeMap(&ma, A, (uint64_t)M, (uint64_t)K, HALF)); else DFCHECK(gemmMakeMap(&ma, A, (uint64_t)K, (uint64_t)M, BK));
  if (!bMn) DFCHECK(gemmMakeMap(&mb, B, (uint64_t)N, (uint64_t)K, HALF)); else DFCHECK(gemmMakeMap(&mb, B, (uint64_t)K, (uint64_t)N, BK));
  CUDACHECK(allowPairs());
  PairArgs g;
  memset(&g, 0, sizeof(g));
  g.C = (__nv_bfloat16*)C; g.M = M; g.N = N; g.K = K; g.ldc = N; g.aMn = aMn ? 1 : 0; g.bMn = bMn ? 1 : 0;
  g.err = errDev; g.errHost = errHost;
  if (e) g.e = *e;
  g.wide = (((uintptr_t)C | (uintptr_t)g.e.aux | (uintptr_t)g.e.pre) & 31) == 0;
  { int64_t gm = paramI64("GEMM_RASTER_GROUP", 8); g.groupM = (int)(gm < 1 ? 1 : gm > 64 ? 64 : gm); }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (M + PM - 1) / PM * (N / PN);
  const int pairs = std::min(tiles, maxResidentPairs(dev, sms));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(2 * pairs); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization; at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  CUDACHECK(cudaLaunchKernelEx(&cfg, pairKernel(g.e.kind), ma, mb, g));
  return ncclSuccess;
}

}  // namespace dfccl
