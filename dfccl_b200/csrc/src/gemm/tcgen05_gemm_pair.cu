// bf16 GEMM on CTA pairs (tcgen05 cta_group::2), hand-written for sm_100a:
//     C[M,N] = A[M,K] * B[N,K]^T,  tiles of 256 x tn, one tile per pair of CTAs (a cluster of two SMs) at a time; tn is chosen per
// product, 64 to 256 in steps of 32, from 128 on where B is stored MN-major.  Rows and columns of the last tiles beyond M (a
// multiple of 128) and N are loaded as zeros and not stored.
// Each CTA of a pair loads 128 rows of A and tn / 2 rows of B per stage (64 or 128 of the contraction), the leader's single MMA thread issues
// 256 x tn x 16 instructions that read both CTAs' shared memory, and each CTA ends up with its 128 rows of the accumulator
// in its own tensor memory.  The tensor cores of an SM thus see every B row once per pair instead of once per CTA: half the
// shared-memory operand traffic per FLOP, which is what bounds a one-CTA kernel.
// The width of a tile is what fits the number of tiles to the number of pairs: 3072 x 1024 outputs are 48 tiles of 256 x 256
// on 74 pairs, or 72 of 256 x 192.
//
// Roles per CTA: warp 0 = TMA producer (one elected thread; completion of both CTAs' loads is counted on the
// LEADER's barrier), warp 1 = tensor-memory owner, and in the leader the MMA issuer; the other warps = epilogue over the
// CTA's own accumulator half, 32 rows x 32 columns at a time: tensor memory -> registers -> global memory, through boxes in
// shared memory and TMA stores where the epilogue is what a tile waits for (gemmPairLaunch).
// Stages are released and accumulators handed over with tcgen05.commit to both CTAs;
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

constexpr int PM = 256, HALF = 128, MAX_STAGES = 6, UMMA_K = 16;
constexpr int SMEM_LIMIT = 227 * 1024, BAR_BYTES = 256, ALIGN_SLACK = 1024;
constexpr int BOX_BYTES = 32 * 64;                   // a staged box of the epilogue: 32 rows x 32 columns
constexpr int EPI_BOXES = 16, EPI_BYTES = EPI_BOXES * BOX_BYTES;      // boxes of their own, where a pair has several tiles
constexpr int WIDE_STAGE = (HALF + 128) * 64 * 2;    // a stage of the widest tile, per CTA
constexpr uint64_t WAIT_NS = 4000000000ull;          // nothing here waits on another GPU: seconds mean a lost partner

// Epilogue warps: two per 32 accumulator rows, four where an element costs more than its rounding (8192 x 4096 x 1024 with bias and
// residual 63 -> 59.7 us, with GELU 63.3 -> 60.3, with its gradient 71 -> 67.9; plain small products lose 0.3 - 0.5 us with four).
__host__ __device__ constexpr int epiWarps(int epi) { return epi == EPI_NONE || epi == EPI_BIAS ? 8 : 16; }
__host__ __device__ constexpr int pairThreads(int epi) { return 64 + 32 * epiWarps(epi); }

// A stage: `kSteps` blocks of 64 of the contraction (gemmPairLaunch), HALF rows of A and half the tile's columns of B.
constexpr int kSteps(int width) { return width >= 224 ? 1 : 2; }
constexpr int bBytesOf(int width, bool bMn) { return (bMn ? (width / 2 + 63) / 64 * 64 : width / 2) * 64 * kSteps(width) * 2; }
constexpr int stageBytesOf(int width, bool bMn) { return HALF * 64 * kSteps(width) * 2 + bBytesOf(width, bMn); }
// Boxes of one epilogue warp where a pair has one tile, and the stages that hold all of them.
constexpr int boxesOnce(int epi, int width, bool stored) { return (width / 32 + epiWarps(epi) / 4 - 1) / (epiWarps(epi) / 4) * (stored ? 2 : 1); }
constexpr int stagesOnce(int epi, int width, bool bMn, bool stored) {
  return (epiWarps(epi) * boxesOnce(epi, width, stored) * BOX_BYTES + stageBytesOf(width, bMn) - 1) / stageBytesOf(width, bMn);
}
// They have a barrier each and fit in front of the barriers: five stages (150 KB) at width 224 and three of 56 KB at 192, with GELU and
// its pre-activation stored, are the most.
constexpr bool boxesFit() {
  for (int epi = EPI_NONE; epi <= EPI_GELU_GRAD; ++epi)
    for (int width = 64; width <= 256; width += 32)
      for (int i = 0; i < 4; ++i) {
        const int stages = stagesOnce(epi, width, (i & 1) != 0, i >= 2 && epi == EPI_BIAS_GELU);
        if (stages > MAX_STAGES || stages * stageBytesOf(width, (i & 1) != 0) > SMEM_LIMIT - BAR_BYTES - ALIGN_SLACK) return false;
      }
  return true;
}
static_assert(boxesFit(), "the boxes of a pair's only tile do not fit its operands' stages");

struct PairArgs {
  int M, N, K, ldc;
  int aMn, bMn;
  int tn;                           // columns of a tile
  int kStep;                        // blocks of 64 of the contraction in a stage: 1 or 2
  int stages, stageBytes;
  int tmemCols;                     // 512: two accumulators at columns 0 and 256; less: one, and no pair has a second tile
  int groupM;                       // row tiles per rasterisation group
  uint32_t* err;
  uint32_t* errHost;
  __nv_bfloat16* C;
  GemmEpilogue e;
  bool boxes;                       // results go through boxes (the kinds without a choice: GELU_GRAD never, others always)
  int once;                         // a pair has one tile: the boxes of one of its warps, in the operands' stages; 0: several, boxes of their own
  int epiBytes;                     // of those
  bool wide, wideC;                 // aux, and C and pre, start on a 32-byte boundary
};

// WIDE: tiles of 256 x 256 in stages of 64, known to the compiler: the loops that issue loads and MMAs keep no geometry.  us:
// 8192 x 4096 x 1024 56.0 -> 55.6, its data gradient 56.2 -> 55.7, 4096 x 4096 x 1024 and its gradients 94.0 -> 93.8.
template <int EPI, bool WIDE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pairThreads(EPI), 1)
dfcclGemmPairKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const __grid_constant__ CUtensorMap mapC,
                    const __grid_constant__ CUtensorMap mapPre, const PairArgs g) {
  const int tn = WIDE ? 256 : g.tn, kStep = WIDE ? 1 : g.kStep, stageBytes = WIDE ? WIDE_STAGE : g.stageBytes;
  constexpr int EPI_WARPS = epiWarps(EPI), PARTS = EPI_WARPS / 4, BUFS = EPI_BOXES / EPI_WARPS;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);       // the same offset in both CTAs
  uint8_t* stg = smem + g.stages * stageBytes;
  uint64_t* fullBar = (uint64_t*)(stg + g.epiBytes);                  // used in the leader only
  uint64_t* emptyBar = fullBar + MAX_STAGES;                         // in both CTAs (commit to both)
  uint64_t* accFull = emptyBar + MAX_STAGES;                         // [2] in both CTAs
  uint64_t* accEmpty = accFull + 2;                                  // [2] used in the leader only: the epilogue warps of both CTAs arrive
  uint32_t* tmemBaseSlot = (uint32_t*)(accEmpty + 2);
  volatile uint32_t* giveUp = tmemBaseSlot + 1;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t cr = cluster_ctarank();             // 0 = leader
  const int mTiles = (g.M + PM - 1) / PM, nTiles = (g.N + tn - 1) / tn, kb64 = g.K / 64;
  const int numTiles = mTiles * nTiles;
  const int pair = blockIdx.x >> 1, numPairs = gridDim.x >> 1;
  const int bHalf = tn / 2;
  const int aBytes = HALF * 128 * kStep, mnBlock = 64 * 128 * kStep;      // MN-major operand: blocks of 64 MN-columns x K-rows; K-major: 64 K-columns x rows

  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) { mbar_init(&fullBar[s], 1); mbar_init(&emptyBar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&accFull[a], 1); mbar_init(&accEmpty[a], 2 * EPI_WARPS); }
    // (not the device's error word: read here, beside the kernel in front, it could differ between the two CTAs, and one would
    // wait for a partner that does nothing.  After a kernel has given up the host refuses launches.)
    *giveUp = 0;
    mbar_fence_init();
    tma_prefetch_desc(&mapA);
    tma_prefetch_desc(&mapB);
    if (g.boxes) tma_prefetch_desc(&mapC);
  }
  if (warp == 1) tmem_alloc_pair(tmemBaseSlot, g.tmemCols);
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
      // One load per operand and stage where it is cut into whole blocks of 64 columns or rows: K-major operand [rows, K] as
      // (64 K, rows, K / 64), boxes of 64 x rows x kStep; MN-major operand [K, cols] as (64 cols, K, cols / 64), boxes of
      // 64 x 64 kStep x (cols / 64).  An MN-major B whose tiles are not whole blocks is loaded block by block, from any multiple
      // of 16 columns.  The second half of the last stage may lie outside (zeros): it is loaded and not multiplied.
      const uint32_t bar0 = mapa_u32(smem_u32(fullBar), 0);
      const bool bLoose = !WIDE && g.bMn && bHalf % 64 != 0;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += numPairs) {
        int mt, nt;
        raster_tile(t, mTiles, nTiles, g.groupM, mt, nt);
        const int rowA = mt * PM + (int)cr * HALF, rowB = nt * tn + (int)cr * bHalf;
        for (int k = 0; k < kb64; k += kStep) {
          if (!mbar_wait(&emptyBar[stage], phase ^ 1, giveUp, WAIT_NS)) { ok = false; break; }
          if (cr == 0) mbar_expect_tx(&fullBar[stage], 2 * stageBytes);       // my bytes and the partner's
          uint8_t* sa = smem + stage * stageBytes;
          const uint32_t bar = bar0 + stage * 8;
          tma_load_3d_pair(sa, &mapA, g.aMn ? k * 64 : rowA, g.aMn ? rowA / 64 : k, bar);
          if (!bLoose) tma_load_3d_pair(sa + aBytes, &mapB, g.bMn ? k * 64 : rowB, g.bMn ? rowB / 64 : k, bar);
          else for (int i = 0; i * 64 < bHalf; ++i) tma_load_2d_pair(sa + aBytes + i * mnBlock, &mapB, rowB + 64 * i, k * 64, bar);
          if (++stage == g.stages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) for (int i = 0; i < 20000; ++i) __nanosleep(200);     // copies already issued land before the CTA goes away
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (cr == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(PM, tn, g.aMn, g.bMn);
      // per instruction (16 K): K-major 32 bytes along the row; MN-major two groups of 8 K-rows.  Per 64 K: the next block of
      // [rows] x 64 K-columns, or 64 K-rows further down the same blocks.
      const uint32_t stepA = g.aMn ? 128u : 2u, stepB = g.bMn ? 128u : 2u;
      const uint32_t hopA = g.aMn ? 512u : HALF * 128 / 16, hopB = g.bMn ? 512u : (uint32_t)bHalf * 128 / 16;
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      int loads = (numTiles - pair + numPairs - 1) / numPairs * ((kb64 + kStep - 1) / kStep) - g.stages;     // that wait for a stage
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += numPairs, ++it) {
        const int ab = it & 1;
        if (!mbar_wait(&accEmpty[ab], ((it >> 1) & 1) ^ 1, giveUp, WAIT_NS)) break;
        tc_fence_after();
        const uint32_t d = tmemBase + ab * 256;
        for (int kb = 0; kb < kb64; kb += kStep) {
          if (!mbar_wait(&fullBar[stage], phase, giveUp, WAIT_NS)) { ok = false; break; }
          tc_fence_after();
          const uint8_t* pa = smem + stage * stageBytes;
          const uint64_t da = g.aMn ? umma_smem_desc_mn_sw128(pa, mnBlock) : umma_smem_desc_sw128(pa);
          const uint64_t db = g.bMn ? umma_smem_desc_mn_sw128(pa + aBytes, mnBlock) : umma_smem_desc_sw128(pa + aBytes);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h == 1 && (kStep == 1 || kb + 1 == kb64)) break;
#pragma unroll
            for (int k = 0; k < 64 / UMMA_K; ++k)
              umma_bf16_pair(d, da + hopA * h + stepA * k, db + hopB * h + stepB * k, idesc, (kb | h | k) != 0);
          }
          if (loads-- > 0) umma_commit_pair(&emptyBar[stage]);      // both CTAs' stage is free once these MMAs have read it
          if (++stage == g.stages) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit_pair(&accFull[ab]);       // both halves of the accumulator complete
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: my 128 rows, TMEM -> bf16 -> boxes -> global
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const uint32_t accEmptyLeader0 = mapa_u32(smem_u32(&accEmpty[0]), 0), accEmptyLeader1 = mapa_u32(smem_u32(&accEmpty[1]), 0);
    // A box is stored with the 64-byte swizzle: 16-byte chunk c of row r sits at chunk c ^ (r / 2 % 4), so that eight lanes
    // (rows) that write the same chunk meet eight different groups of four banks.
    // A pair's only tile finds the operands' stages free, with a box for every store: none waits for another one's.
    uint8_t* const box0 = g.once ? smem + (warp - 2) * g.once * BOX_BYTES : stg + (warp - 2) * BUFS * BOX_BYTES;
    const uint32_t rowOff = lane * 64, swz = (lane >> 1) & 3;
    int turn = 0;
    auto store = [&](const CUtensorMap* map, __nv_bfloat16* base, const uint4 (&o)[4], int x, int y) {
      if (EPI == EPI_GELU_GRAD || ((EPI == EPI_NONE || EPI == EPI_BIAS) && !g.boxes)) {      // 64 bytes of its row per lane, in whole sectors
        __nv_bfloat16* p = base + (size_t)(y + lane) * g.ldc + x;
        st_global32(p, o, g.wideC);
        st_global32(p + 16, o + 2, g.wideC);
        return;
      }
      uint8_t* box = box0 + turn * BOX_BYTES;
      if (!g.once) {
        if (lane == 0) bulk_wait_read<BUFS - 1>();     // the store that read this buffer last has done so
        __syncwarp();
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) *(uint4*)(box + rowOff + ((v ^ swz) << 4)) = o[v];
      fence_async_shared();
      __syncwarp();
      if (lane == 0) { tma_store_2d(map, box, x, y); bulk_commit(); }
      if (++turn == BUFS && !g.once) turn = 0;
    };
    int it = 0;
    for (int t = pair; t < numTiles; t += numPairs, ++it) {
      int mt, nt;
      raster_tile(t, mTiles, nTiles, g.groupM, mt, nt);
      const int ab = it & 1;
      const int row0 = mt * PM + (int)cr * HALF + quarter * 32, col0 = nt * tn;      // of this warp's 32 rows
      const bool mine = row0 < g.M;                                   // the last row tile may have only its upper half
      const int steps = min(tn, g.N - col0) / 32;
      constexpr bool AUX = EPI == EPI_BIAS_RES || EPI == EPI_GELU_GRAD;
      const __nv_bfloat16* aux = g.e.aux + (size_t)(row0 + lane) * g.ldc + col0;
      uint4 own[4];
      auto loadAux = [&](int i) {
        if (!AUX || !mine || i >= steps) return;
        ld_global32(aux + i * 32, own, g.wide);
        ld_global32(aux + i * 32 + 16, own + 2, g.wide);
      };
      constexpr bool AHEAD = EPI == EPI_BIAS_RES;      // (GELU's gradient needs the registers)
      if (AHEAD) loadAux(part);                        // on its way while the accumulator is computed
      if (!mbar_wait(&accFull[ab], (it >> 1) & 1, giveUp, WAIT_NS)) break;
      tc_fence_after();
#pragma unroll 1
      for (int i = part; i < steps; i += PARTS) {
        if (!mine) break;
        const int c = i * 32;
        uint32_t r[32];
        tmem_ld32(tmemBase + ((uint32_t)(quarter * 32) << 16) + ab * 256 + c, r);
        if (!AHEAD) loadAux(i);
        tmem_ld_wait();
        if (EPI == EPI_BIAS || EPI == EPI_BIAS_RES || EPI == EPI_BIAS_GELU) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const uint4 bv = ((const uint4*)(g.e.bias + col0 + c))[v];
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
          if (AHEAD) loadAux(i + PARTS);
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
          if (g.e.pre) store(&mapPre, g.e.pre, o, col0 + c, row0);
#pragma unroll
          for (int v = 0; v < 4; ++v) {                // of the rounded value: what the backward pass differentiates at
            uint32_t* ow = (uint32_t*)&o[v];
#pragma unroll
            for (int w = 0; w < 4; ++w) ow[w] = pack_bf16x2(geluTanh(bf16Lo(ow[w])), geluTanh(bf16Hi(ow[w])));
          }
        }
        store(&mapC, g.C, o, col0 + c, row0);
      }
      if (t + 2 * numPairs < numTiles) {               // the pair's epilogue warps release the accumulator to the tile after the next
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(ab ? accEmptyLeader1 : accEmptyLeader0);
      }
    }
    if (lane == 0) bulk_wait_read<0>();                // the boxes have been read before the CTA's shared memory goes away
  }

  // ---------------------------------------------------------------- leave: nothing of the pair may still use my shared or tensor memory
  // (Every arrival between the CTAs is one that somebody has waited for, so that none is on its way any more; and none of them, nor the
  // barrier, waits for the epilogue's stores, which the end of the kernel does anyway.  With releasing arrivals, one for every accumulator,
  // a CTA left 1.3 us after its last store.)
  tc_fence_before();
  __syncthreads();
  cluster_sync_relaxed();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmemBase, g.tmemCols);
  if (threadIdx.x == 0 && *giveUp) { atomicExch(g.err, 1u); *(volatile uint32_t*)g.errHost = 1u; __threadfence_system(); }
}

}  // namespace

namespace {
typedef void (*PairKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const PairArgs);
template <bool WIDE>
PairKernel pairKernelOf(int epi) {
  static const PairKernel k[] = {dfcclGemmPairKernel<EPI_NONE, WIDE>, dfcclGemmPairKernel<EPI_BIAS, WIDE>, dfcclGemmPairKernel<EPI_BIAS_RES, WIDE>,
                                 dfcclGemmPairKernel<EPI_BIAS_GELU, WIDE>, dfcclGemmPairKernel<EPI_GELU_GRAD, WIDE>};
  return k[epi];
}
PairKernel pairKernel(int epi, bool wide) { return wide ? pairKernelOf<true>(epi) : pairKernelOf<false>(epi); }
cudaError_t allowPairs() {
  return oncePerDevice([] {
    cudaError_t r = cudaSuccess;
    for (int e = EPI_NONE; e <= EPI_GELU_GRAD; ++e)
      for (int w = 0; w < 2 && r == cudaSuccess; ++w) r = allowSharedMemory(pairKernel(e, w != 0), SMEM_LIMIT);
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
    cfg.gridDim = dim3(sms & ~1); cfg.blockDim = dim3(pairThreads(EPI_NONE)); cfg.dynamicSmemBytes = SMEM_LIMIT;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, pairKernel(EPI_NONE, true), &cfg) != cudaSuccess || n <= 0) { (void)cudaGetLastError(); n = sms / 2; }
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

ncclResult_t gemmPairLaunch(int width, const void* A, const void* B, void* C, int M, int N, int K, cudaStream_t stream, int aMn, int bMn,
                            uint32_t* errDev, uint32_t* errHost, const GemmEpilogue* e) {
  CUDACHECK(allowPairs());
  // 64 of the contraction in a stage keep more loads in flight beside wide tiles (stages of 128: 8192 x 4096 x 1024 and its
  // gradients 0.3 - 0.5 % slower, 4096 x 1024 x 8192 the same); for narrower ones the tensor cores are through with such a stage
  // before its two loads are issued (460 clocks)
  const int kStep = kSteps(width), BK = 64 * kStep, bHalf = width / 2;
  CUtensorMap ma, mb, mc, mp;
  DFCHECK(gemmMakeMap3(&ma, A, (uint64_t)M, (uint64_t)K, aMn, HALF, BK));
  if (bMn && bHalf % 64) DFCHECK(gemmMakeMap(&mb, B, (uint64_t)K, (uint64_t)N, BK));
  else DFCHECK(gemmMakeMap3(&mb, B, (uint64_t)N, (uint64_t)K, bMn, bHalf, BK));
  PairArgs g;
  memset(&g, 0, sizeof(g));
  g.M = M; g.N = N; g.K = K; g.ldc = N; g.aMn = aMn ? 1 : 0; g.bMn = bMn ? 1 : 0; g.tn = width;
  g.err = errDev; g.errHost = errHost;
  if (e) g.e = *e;
  g.C = (__nv_bfloat16*)C;
  g.wide = ((uintptr_t)g.e.aux & 31) == 0;
  g.wideC = (((uintptr_t)C | (uintptr_t)g.e.pre) & 31) == 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (M + PM - 1) / PM * ((N + width - 1) / width);
  const int pairs = std::min(tiles, maxResidentPairs(dev, sms));
  // Boxes and TMA stores drain a tile faster, straight stores leave the loads' engine and 32 KB of stages to the operands of the tiles
  // that follow: a pair's only tile, whose boxes lie in the stages it no longer needs, goes through them, others with short
  // contractions.  us, boxes / straight: 1920 x 1792 x 3072 18.0 / 18.6, 3200 x 768 x 1088 11.4 / 11.7; several tiles, widths from 224 on: up to
  // K = 256 14 % less with boxes, 512 4 %, 768 the same, 1024 1 % more, 1536 2 %; narrower ones 8 %, 0, 2 % more, 3 %, 4 % (230 and 800
  // products of all storage orders).  A bias, added between tensor memory and the store, moves the line of the wide ones: 8192 x 4096 x
  // 768 44.9 / 47.9, x 832 46.1 / 47.8, x 896 48.7 / 49.5, x 1024 56.5 / 57.2, 5376 x 4096 x 768 29.4 / 30.9, x 896 35.3 / 36.1, 4096 x 3072 x 768 17.8 /
  // 18.7, x 896 22.1 / 22.3, x 1024 23.9 / 23.8, 16384 x 768 x 768 19.6 / 20.2, x 896 23.4 / 23.7, x 1024 25.7 / 25.6, 3840 x 1792 x 896 14.2 / 14.0; not that of
  // narrower ones: 2560 x 3840 x 512 13.5 / 13.7, x 768 16.6 / 15.2, 2176 x 2304 x 768 11.9 / 10.7, x 1024 13.2 / 12.0.
  const int line = g.e.kind == EPI_BIAS && width >= 224 ? 1024 : 768;
  const bool straight = g.e.kind == EPI_GELU_GRAD || ((g.e.kind == EPI_NONE || g.e.kind == EPI_BIAS) && tiles > pairs && K >= line);
  const bool stored = g.e.kind == EPI_BIAS_GELU && g.e.pre;
  g.boxes = !straight;
  g.once = tiles > pairs ? 0 : boxesOnce(g.e.kind, width, stored);
  g.epiBytes = g.boxes && !g.once ? EPI_BYTES : 0;
  mc = ma;                                             // (straight stores take no map: none is made, or kept, per output)
  if (!straight) DFCHECK(gemmMakeMap(&mc, C, (uint64_t)M, (uint64_t)N, 32, 32));
  mp = mc;
  if (g.e.kind == EPI_BIAS_GELU && g.e.pre) DFCHECK(gemmMakeMap(&mp, g.e.pre, (uint64_t)M, (uint64_t)N, 32, 32));
  // (where every pair has one tile the order decides nothing)
  { int64_t gm = tiles > pairs ? paramI64("GEMM_RASTER_GROUP", 8) : 8; g.groupM = (int)(gm < 1 ? 1 : gm > 64 ? 64 : gm); }
  g.kStep = kStep;
  g.stageBytes = stageBytesOf(width, bMn != 0);        // width 256: WIDE_STAGE, however B is stored
  const int room = SMEM_LIMIT - BAR_BYTES - ALIGN_SLACK - g.epiBytes;
  const int want = tiles > pairs ? MAX_STAGES : (K + BK - 1) / BK;
  g.stages = std::min(std::min(MAX_STAGES, room / g.stageBytes), want);
  if (g.boxes && g.once) g.stages = std::max(g.stages, stagesOnce(g.e.kind, width, bMn != 0, stored));        // (boxesFit)
  if (g.stages > MAX_STAGES || g.stages * g.stageBytes > room) return ncclInternalError;
  g.tmemCols = tiles > pairs ? 512 : width <= 64 ? 64 : width <= 128 ? 128 : 256;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(2 * pairs); cfg.blockDim = dim3(pairThreads(g.e.kind)); cfg.stream = stream;
  // at least the SM's shared memory times the share of its tensor memory: CTAs that are resident together, of this launch, of
  // the next one or of another stream, then never wait for tensor memory
  cfg.dynamicSmemBytes = std::max(g.stages * g.stageBytes + g.epiBytes + BAR_BYTES + ALIGN_SLACK, 228 * 1024 * g.tmemCols / 512 - 1024);
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization; at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  CUDACHECK(cudaLaunchKernelEx(&cfg, pairKernel(g.e.kind, width == 256), ma, mb, mc, mp, g));
  return ncclSuccess;
}

}  // namespace dfccl
