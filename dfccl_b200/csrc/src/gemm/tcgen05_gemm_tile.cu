// bf16 GEMM for products too small to fill the GPU with tiles of 256 x 256, hand-written for sm_100a:
//     C[M,N] = A[M,K] * B[N,K]^T, one tile (or one slice of a tile's contraction) per CTA or CTA pair.
//
// What bounds such a product is how few SMs a handful of tiles occupies, the issue of loads and MMAs in a CTA (about 80 clocks
// per MMA of 16 K however narrow the tile, 230 per load instruction: hence 128 K and one load per operand in a stage),
// and the fixed cost of a launch.
//   * Tiles of 128 x {64, 128} on one CTA (cta_group::1) or 256 x {128, 256} on a pair (cta_group::2, each CTA loads
//     half of B: fewer operand bytes per FLOP); the last row tile may stick out of M (TMA fills zeros, rows are not stored).
//   * The contraction of a tile is cut into up to 4 slices on the CTAs of one cluster.  Every CTA of the cluster owns
//     a slice of the tile's columns: the others write their fp32 partial sums of those columns into the owner's shared
//     memory (distributed shared memory), the owner adds them in slice order and stores bf16.  No workspace in global
//     memory, no second kernel, no atomics: the result does not depend on timing.
//   * Programmatic dependent launch: barriers, tensor memory and descriptors of a launch are set up while the kernel in
//     front of it in the stream still runs; nothing is read or written before griddepcontrol.wait.
// Which tile and how many slices: gemmTilePlan below.  Measured against the persistent kernels before it (back to back
// in a graph, us): see the table at the plan.
//
// Roles per CTA: warp 0 = TMA producer, warp 1 = tensor-memory owner and (in the leader of a pair) MMA issuer, warps 2-9 =
// epilogue, two warps per 32 accumulator rows.  No TMA load uses cluster multicast; every wait is bounded.
#include "tc_common.h"
#include "gemm.h"
#include "../common/device_once.h"
#include "../common/log.h"
#include <algorithm>

namespace dfccl {
namespace {

using namespace tc;

constexpr int TM = 128, BK = 128, UMMA_K = 16, MAX_STAGES = 4;
constexpr int A_BYTES = TM * BK * 2;
constexpr int MN_BLOCK_BYTES = 64 * BK * 2;          // MN-major operand: 64 MN-columns x BK K-rows; K-major: 64 K-columns x rows
constexpr int NUM_THREADS = 320;                     // 10 warps
constexpr int EPI_ROW_BYTES = 64 * 2 + 16;           // a staged row of the epilogue: rows start in different banks
constexpr int EPI_BYTES = 8 * 32 * EPI_ROW_BYTES;    // one buffer of 32 rows per epilogue warp, in the operands' stages once those are done
constexpr int BOX_BYTES = 32 * 64;                   // whole contractions: boxes of 32 rows x 32 columns, in the same place
constexpr int SMEM_LIMIT = 227 * 1024, BAR_BYTES = 256, ALIGN_SLACK = 1024;
constexpr uint64_t WAIT_NS = 4000000000ull;          // nothing here waits on another GPU: seconds mean a lost partner

struct TileArgs {
  __nv_bfloat16* C;
  int M, N, K;
  int aMn, bMn;
  int split;                        // slices of the contraction = CTAs (pairs) of a tile
  int stages;
  uint32_t* err;
  uint32_t* errHost;
};

__host__ __device__ constexpr int bRows(bool pair, int tn) { return pair ? tn / 2 : tn; }                    // rows of B a CTA loads per K block
__host__ __device__ constexpr int stageBytes(bool pair, int tn) { return A_BYTES + bRows(pair, tn) * BK * 2; }
// Whole contractions leave through boxes and TMA stores where a warp has two blocks of 32 columns or more.  us, row segments / boxes:
// 4096 x 1024 x 1024 (tiles of 256 x 256) 10.4 / 9.9, 1920 x 1792 x 3072 19.8 / 19.4, 512 x 4096 x 768 (256 x 128) 6.15 / 6.04, 2944 x 512 x
// 256 (128 x 128) 5.84 / 5.73; but 768 x 1024 x 512 (128 x 64) 4.81 / 4.92.
__host__ __device__ constexpr bool boxed(int tn) { return tn >= 128; }
__host__ __device__ constexpr int exchangeBytes(int tn, int split) { return split > 1 ? (split - 1) * TM * (tn / split) * 4 : 0; }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void st_cluster16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

template <bool PAIR, int TN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
dfcclGemmTileKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const __grid_constant__ CUtensorMap mapC,
                    const TileArgs g) {
  constexpr int STAGE_BYTES = stageBytes(PAIR, TN), BROWS = bRows(PAIR, TN);
  constexpr bool BOXED = boxed(TN);
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);       // the same offset in every CTA of the cluster
  uint8_t* exch = smem + max(g.stages * STAGE_BYTES, EPI_BYTES);                                // [split - 1][columns / 4][128 rows] of 16 bytes
  uint64_t* fullBar = (uint64_t*)(exch + exchangeBytes(TN, g.split));               // pair: used in the leader only
  uint64_t* emptyBar = fullBar + MAX_STAGES;
  uint64_t* accFull = emptyBar + MAX_STAGES;
  uint32_t* tmemBaseSlot = (uint32_t*)(accFull + 1);
  volatile uint32_t* giveUp = tmemBaseSlot + 1;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int clusterSize = (PAIR ? 2 : 1) * g.split;
  const uint32_t cr = clusterSize > 1 ? cluster_ctarank() : 0;
  const uint32_t half = PAIR ? cr & 1 : 0, leader = cr - half;                      // my half of a pair's rows; the pair's first CTA
  const int slice = PAIR ? (int)(cr >> 1) : (int)cr;
  const int tile = blockIdx.x / clusterSize;
  const int nTiles = g.N / TN;
  const int mt = tile / nTiles, nt = tile - mt * nTiles;
  const int kb64 = g.K / 64;
  const int k0 = slice * kb64 / g.split, k1 = (slice + 1) * kb64 / g.split;        // my blocks of 64 of the contraction: never none, split <= K / 64
  const int rowBase = (PAIR ? mt * 2 + (int)half : mt) * TM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) { mbar_init(&fullBar[s], 1); mbar_init(&emptyBar[s], 1); }
    mbar_init(accFull, 1);
    *giveUp = 0;
    mbar_fence_init();
    tma_prefetch_desc(&mapA);
    tma_prefetch_desc(&mapB);
    if (BOXED && g.split == 1) tma_prefetch_desc(&mapC);
  }
  if (warp == 1) { if (PAIR) tmem_alloc_pair(tmemBaseSlot, TN); else tmem_alloc(tmemBaseSlot, TN); }
  tc_fence_before();
  __syncthreads();
  if (clusterSize > 1) cluster_sync_all();           // the other CTAs' barriers and shared memory exist
  tc_fence_after();
  const uint32_t tmemBase = *tmemBaseSlot;
  grid_dependency_wait();                            // everything above may run beside the kernel in front of this one
  grid_launch_dependents();

  if (warp == 0) {
    if (elect_one()) {
      // One load per operand and stage.  K-major operand [rows, K] as (64 K, rows, K / 64), boxes of 64 x rows x 2; MN-major
      // operand [K, cols] as (64 cols, K, cols / 64), boxes of 64 x 128 x (rows / 64).  The second half of the last stage
      // of a slice may belong to the next slice or lie outside (zeros): it is loaded and not multiplied.
      const uint32_t bar0 = PAIR ? mapa_u32(smem_u32(fullBar), leader) : 0;
      const int rowB = nt * TN + (int)half * BROWS;
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int k = k0; k < k1; k += 2) {
        if (!mbar_wait(&emptyBar[stage], phase ^ 1, giveUp, WAIT_NS)) { ok = false; break; }
        if (half == 0) mbar_expect_tx(&fullBar[stage], (PAIR ? 2 : 1) * STAGE_BYTES);
        uint8_t* sa = smem + stage * STAGE_BYTES;
        const int ya = g.aMn ? k * 64 : rowBase, za = g.aMn ? rowBase / 64 : k;
        const int yb = g.bMn ? k * 64 : rowB, zb = g.bMn ? rowB / 64 : k;
        if (PAIR) {
          tma_load_3d_pair(sa, &mapA, ya, za, bar0 + stage * 8);
          tma_load_3d_pair(sa + A_BYTES, &mapB, yb, zb, bar0 + stage * 8);
        } else {
          tma_load_3d(sa, &mapA, ya, za, &fullBar[stage]);
          tma_load_3d(sa + A_BYTES, &mapB, yb, zb, &fullBar[stage]);
        }
        if (++stage == g.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok) for (int i = 0; i < 20000; ++i) __nanosleep(200);     // copies already issued land before the CTA goes away
    }
  } else if (warp == 1) {
    if (half == 0 && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(PAIR ? 2 * TM : TM, TN, g.aMn, g.bMn);
      // per instruction (16 K): K-major 32 bytes along the row; MN-major two groups of 8 K-rows.  Per 64 K: the next block of
      // [rows] x 64 K-columns, or 64 K-rows further down the same blocks.
      const uint32_t stepA = g.aMn ? 128u : 2u, stepB = g.bMn ? 128u : 2u;
      const uint32_t hopA = g.aMn ? 512u : TM * 128 / 16, hopB = g.bMn ? 512u : BROWS * 128 / 16;
      const uint16_t mask = (uint16_t)(3u << leader);
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int k = k0; k < k1; k += 2) {
        if (!mbar_wait(&fullBar[stage], phase, giveUp, WAIT_NS)) { ok = false; break; }
        tc_fence_after();
        const uint8_t* pa = smem + stage * STAGE_BYTES;
        const uint64_t da = g.aMn ? umma_smem_desc_mn_sw128(pa, MN_BLOCK_BYTES) : umma_smem_desc_sw128(pa);
        const uint64_t db = g.bMn ? umma_smem_desc_mn_sw128(pa + A_BYTES, MN_BLOCK_BYTES) : umma_smem_desc_sw128(pa + A_BYTES);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h == 1 && k + 1 == k1) break;
#pragma unroll
          for (int i = 0; i < 64 / UMMA_K; ++i) {
            const uint64_t dai = da + hopA * h + stepA * i, dbi = db + hopB * h + stepB * i;
            if (PAIR) umma_bf16_pair(tmemBase, dai, dbi, idesc, (k > k0) | (h | i));
            else umma_bf16(tmemBase, dai, dbi, idesc, (k > k0) | (h | i));
          }
        }
        if (k + 2 * g.stages < k1) {                  // (a load waits for the stage)
          if (PAIR) umma_commit_pair(&emptyBar[stage], mask); else umma_commit(&emptyBar[stage]);
        }
        if (++stage == g.stages) { stage = 0; phase ^= 1; }
      }
      if (ok) { if (PAIR) umma_commit_pair(accFull, mask); else umma_commit(accFull); }
    }
  }

  // ---------------------------------------------------------------- epilogue: two warps per 32 accumulator rows, half of the columns each
  const int quarter = warp & 3, colHalf = (warp - 2) >> 2;
  const int W = TN / g.split;                                        // columns of the tile I finish
  const uint32_t tRow = tmemBase + ((uint32_t)(quarter * 32) << 16);
  const int row = quarter * 32 + lane;
  bool accOk = false;
  if (warp >= 2) {
    accOk = __all_sync(0xffffffffu, mbar_wait(accFull, 0, giveUp, WAIT_NS));
    tc_fence_after();
  }
  if (BOXED && g.split == 1) {
    // 32 rows x 32 columns at a time: tensor memory -> a box in the operands' stages, which are done with -> a TMA store.  In a box,
    // 16-byte chunk c of row r sits at chunk c ^ (r / 2 % 4) (the 64-byte swizzle): eight lanes that write the same chunk meet
    // eight different groups of four banks.
    if (warp >= 2 && accOk && rowBase < g.M) {
      constexpr int BOXES = TN / 64;
      const uint32_t swz = (lane >> 1) & 3;
#pragma unroll 1
      for (int i = 0; i < BOXES; ++i) {
        const int c = colHalf * (TN / 2) + i * 32;
        uint8_t* box = smem + ((warp - 2) * BOXES + i) * BOX_BYTES;
        uint32_t r[32];
        tmem_ld32(tRow + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(r[8 * v]), __uint_as_float(r[8 * v + 1]));
          o.y = pack_bf16x2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3]));
          o.z = pack_bf16x2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5]));
          o.w = pack_bf16x2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7]));
          *(uint4*)(box + lane * 64 + ((v ^ swz) << 4)) = o;
        }
        fence_async_shared();
        __syncwarp();
        if (lane == 0) { tma_store_2d(&mapC, box, nt * TN + c, rowBase + quarter * 32); bulk_commit(); }
      }
      if (lane == 0) bulk_wait_read<0>();              // the boxes have been read before the CTA's shared memory goes away
    }
  }
  if (g.split > 1) {
    if (warp >= 2 && accOk) {
      for (int c = colHalf * 32; c < TN; c += 64) {
        if (W >= 32 && c / W == slice) continue;
        uint32_t r[32];
        tmem_ld32(tRow + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int p = 0; p < 2; ++p) {                                // 16 columns always have one owner
          const int cc = c + 16 * p, owner = cc / W;
          if (owner == slice) continue;
          const int slot = slice < owner ? slice : slice - 1;        // position of my slice among the owner's partners
          const int chunk = slot * (W / 4) + (cc - owner * W) / 4;
          const uint32_t dst = mapa_u32(smem_u32(exch), PAIR ? 2 * owner + half : owner) + (chunk * TM + row) * 16;
#pragma unroll
          for (int v = 0; v < 4; ++v)
            st_cluster16(dst + v * TM * 16, r[16 * p + 4 * v], r[16 * p + 4 * v + 1], r[16 * p + 4 * v + 2], r[16 * p + 4 * v + 3]);
        }
      }
    }
    __syncwarp();
    cluster_sync_all();                                              // every partial sum is in its owner's shared memory
  }
  if (!(BOXED && g.split == 1) && warp >= 2 && accOk && rowBase < g.M) {          // (whole CTAs only: M and the tiles are multiples of 128)
    // up to 64 columns at a time: tensor memory (+ the partners' sums) -> staging rows -> whole row segments to global memory
    uint8_t* stg = smem + (warp - 2) * 32 * EPI_ROW_BYTES;
    const int cols = max(W / 2, 16), beg = colHalf * cols, step = min(cols, 64), lanesPerRow = step / 8, shift = 31 - __clz(lanesPerRow);
    __nv_bfloat16* cbase = g.C + (size_t)(rowBase + quarter * 32) * g.N + nt * TN + slice * W;
    for (int c = beg; c < min(beg + cols, W); c += step) {              // (16 columns in all: the first warp alone)
      uint32_t r[4][16];
#pragma unroll
      for (int q = 0; q < 4; ++q) if (q * 16 < step) tmem_ld16(tRow + slice * W + c + q * 16, r[q]);
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q * 16 >= step) break;
        float a[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) a[e] = g.split > 1 ? 0.f : __uint_as_float(r[q][e]);
        for (int s = 0; s < g.split && g.split > 1; ++s) {           // in slice order, so that every column sums alike
          if (s == slice) {
#pragma unroll
            for (int e = 0; e < 16; ++e) a[e] += __uint_as_float(r[q][e]);
          } else {
            const float4* src = (const float4*)exch + ((s < slice ? s : s - 1) * (W / 4) + c / 4 + q * 4) * TM + row;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const float4 p = src[v * TM];
              a[4 * v] += p.x; a[4 * v + 1] += p.y; a[4 * v + 2] += p.z; a[4 * v + 3] += p.w;
            }
          }
        }
        uint4* srow = (uint4*)(stg + lane * EPI_ROW_BYTES + q * 32);
        srow[0] = make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7]));
        srow[1] = make_uint4(pack_bf16x2(a[8], a[9]), pack_bf16x2(a[10], a[11]), pack_bf16x2(a[12], a[13]), pack_bf16x2(a[14], a[15]));
      }
      __syncwarp();
      for (int q = 0; q < lanesPerRow; ++q) {
        const int i = q * 32 + lane, rr = i >> shift, cc = i & (lanesPerRow - 1);
        *(uint4*)(cbase + (size_t)rr * g.N + c + cc * 8) = *(const uint4*)(stg + rr * EPI_ROW_BYTES + cc * 16);
      }
      __syncwarp();
    }
  }

  // ---------------------------------------------------------------- leave: nothing of a pair may still use my shared or tensor memory
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_relaxed();                  // (the end of the kernel waits for the stores, the partner need not)
  tc_fence_after();
  if (warp == 1) { if (PAIR) tmem_dealloc_pair(tmemBase, TN); else tmem_dealloc(tmemBase, TN); }
  if (threadIdx.x == 0 && *giveUp) { atomicExch(g.err, 1u); *(volatile uint32_t*)g.errHost = 1u; __threadfence_system(); }
}

typedef void (*TileKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const TileArgs);
TileKernel kernelOf(bool pair, int tn) {
  if (pair) return tn == 128 ? dfcclGemmTileKernel<true, 128> : dfcclGemmTileKernel<true, 256>;
  return tn == 64 ? dfcclGemmTileKernel<false, 64> : dfcclGemmTileKernel<false, 128>;
}

// What a form takes, in us, as measured back to back in a graph: `block` per 64 of the contraction (alone on the GPU; the
// operands' way through L2 adds a fifth when every SM works), `fixed` for everything else of a wave of CTAs.  A block costs
// 128 x 64 about as much as 128 x 128 on a pair's SM, which is why small tiles win only while there are SMs to spare; the
// exchange of partial sums costs about 1 us per 64 columns of the tile, so contractions are cut only where a handful of
// narrow tiles would leave most SMs idle (128 x 256 x 8192: 21.3 us whole, 8.4 us in four slices).
struct Form { bool pair; int tn, split; double block, fixed; };
constexpr Form FORMS[] = {
  {false, 64, 1, 0.150, 2.4}, {false, 64, 2, 0.150, 3.3}, {false, 64, 4, 0.150, 3.6}, {false, 128, 1, 0.172, 2.8},
  {true, 128, 1, 0.140, 3.1}, {true, 128, 2, 0.140, 5.5},
};

int stagesOf(bool pair, int tn, int split, int kBlocks) {
  const int room = SMEM_LIMIT - BAR_BYTES - ALIGN_SLACK - exchangeBytes(tn, split);
  const int longest = (kBlocks + split - 1) / split;                 // blocks of 64 of the longest slice
  return std::min(std::min(MAX_STAGES, room / stageBytes(pair, tn)), (longest + 1) / 2);
}

}  // namespace

// What the whole GPU takes for 64 of the contraction of that many tiles, however they are spread: power, or L2's bandwidth.
double gpuUs(int rows, int tn, int tiles, int sms) { return 0.00156 * tn * tiles * rows / (128.0 * sms); }

// The form with the least expected time: one of those above, or the persistent kernel with tiles of 256 x width.  Whether a
// contraction is cut, and into how many slices, depends on the sizes and on whether there is an epilogue (not on how the operands
// are stored, nor on `pairs`), so that the same product is always summed in the same order; the width of a tile does not change a
// sum.  An epilogue makes whole contractions more frequent (512 x 256 x 1024: four slices without): inside the persistent kernel it
// is applied to the fp32 sum and the result rounded once, behind a cut product to its rounded value.
// The persistent kernel: 3.2 us, and per wave of tiles 0.8 us + per 64 of the contraction what the tensor cores take for
// the width, at least what a CTA's loads take (128 rows of A whatever the width), more when B is stored MN-major
// in blocks of 64 columns that the tiles cut through, and when every SM works; at least what the whole GPU takes for the
// FLOPs.  Fitted to some 500 products of all storage orders at widths of 32 to 256, 5 % rms.
// It overlaps a tile's epilogue with the next tile's loads, the others start anew for every wave, but a wave of them is 0.7 us
// cheaper (smaller blocks, no boxes to drain).  Measured, us (M x N x K: now / the better of these forms and width 256):
//   2176x2304x2048 17.9 / 25.8 (width 160), 1280x3840x2560 21.2 / 29.4 (160), 896x6400x1536 16.9 / 20.1 (192),
//   3072x1024x8192 42.6 / 47.5 (192), 1920x1280x768 7.1 / 8.5 (160), 3072x1792x6528 55.9 / 62.8 (160);
//   a form of one wave: 128x512x512 3.6 (persistent 4.4), 1024x2048x1024 6.8 (7.3), 128x256x8192 8.4 in four slices
//   (whole 21.3).
double pairUs(int M, int N, int kb, int width, int sms, bool bMn) {
  const int pairs = std::max(1, sms / 2), tiles = (M + 255) / 256 * ((N + width - 1) / width), waves = (tiles + pairs - 1) / pairs;
  const double loads = bMn ? 0.13 : 0.092, loose = bMn && width / 2 % 64 ? 0.03 : 0.0;
  const double busy = std::min(1.0, (double)tiles / pairs);
  return 3.2 + waves * 0.8 + kb * std::max(waves * (std::max(loads, 0.00107 * width) + loose + 0.045 * busy), gpuUs(256, width, tiles, sms));
}

static GemmTilePlan choosePlan(int M, int N, int K, int sms, bool pairs, bool bMn, bool epilogue) {
  const int kb = K / 64;
  auto waves = [&](int clusters, int size) {          // clusters of 4 leave SMs of a GPC unused: 36 did not fit
    const int room = size == 1 ? sms : size == 2 ? sms / 2 : sms * 7 / 8 / size;
    return (clusters + std::max(room, 1) - 1) / std::max(room, 1);
  };
  // an epilogue is a pass of its own behind these forms, which reads and writes the product (2048 x 1024: 2.8 us)
  const double pass = epilogue ? 2.3 + 4.0 * M * N / 5e6 : 0.0;
  auto busy = [&](int ctas) { return 1.0 + 0.2 * std::min(1.0, (double)ctas / sms); };
  auto expect = [&](const Form& f) {
    const int size = (f.pair ? 2 : 1) * f.split, rows = f.pair ? 2 * TM : TM;
    const int tiles = (M + rows - 1) / rows * (N / f.tn);
    const int w = waves(tiles, size);
    return w * f.fixed + std::max(w * ((kb + f.split - 1) / f.split * f.block * busy(tiles * size)), kb * gpuUs(rows, f.tn, tiles, sms)) + pass;
  };
  auto best = [&](bool mn, bool whole) {               // `whole`: contractions that are not cut
    GemmTilePlan p{true, 0, 1, 256};
    double us = pairUs(M, N, kb, 256, sms, mn);
    for (int w = mn ? 128 : 64; w < 256; w += 32) {      // (narrower ones never were the least: 780 000 products, 132 and 148 SMs)
      const double t = pairUs(M, N, kb, w, sms, mn);
      if (t < us) { us = t; p.width = w; }
    }
    for (const Form& f : FORMS) {
      if (f.split > kb || (whole && f.split > 1)) continue;
      const double t = expect(f);
      if (t < us) { us = t; p = GemmTilePlan{f.pair, f.tn, f.split, 0}; }
    }
    return p;
  };
  GemmTilePlan p = best(false, false);
  if (p.split == 1 && bMn) p = best(true, true);
  // One wave of plain tiles of 256 x 256 gains nothing from the persistent kernel's overlap, and the form with the same tile has
  // stages of 128 of the contraction and a geometry that the compiler knows.  us, persistent / form: 4096 x 1024 x 8192 58.5 / 56.9,
  // x 2048 16.8 / 15.8, 1024 x 4096 x 8192 59.2 / 57.1, 7168 x 512 x 960 11.9 / 11.3, 3328 x 1024 x 4032 24.4 / 23.8; but 640 x 5120 x 448
  // 7.2 / 7.3, 4096 x 1024 x 128 5.3 / 5.8, and with one or two row tiles, whose operands hardly meet in L2, 512 x 7168 x 4992 29.4 /
  // 31.4, 384 x 7680 x 5248 33.5 / 34.9.  (Before results of either went through boxes in the operands' stages, which brought 4096 x 1024 x
  // 1024 from 10.4 to 9.9 on the form.)
  if (pairs && !epilogue && p.width == 256 && (M + 255) / 256 * (N / 256) <= sms / 2 && K >= 512 && M > 512) p = GemmTilePlan{true, 256, 1, 0};
  if (!pairs && (p.pair || p.width)) {                 // one CTA per tile by request: the same slices
    double us = 1e30;
    const int split = p.split;
    for (const Form& f : FORMS)
      if (!f.pair && f.split == split && expect(f) < us) { us = expect(f); p = GemmTilePlan{f.pair, f.tn, f.split, 0}; }
  }
  return p;
}

// (a product's sizes come back every step: the last few choices of the thread are kept, 0.15 us of a launch)
GemmTilePlan gemmTilePlan(int M, int N, int K, int sms, bool pairs, bool bMn, bool epilogue) {
  struct Kept { int M, N, K, key; GemmTilePlan p; };
  static thread_local Kept kept[64];
  const int key = 1 + sms * 8 + pairs * 4 + bMn * 2 + epilogue;
  Kept& k = kept[((uint32_t)M * 31u + (uint32_t)N * 17u + (uint32_t)K * 7u + (uint32_t)key * 0x9E3779B1u) >> 7 & 63u];
  if (k.key != key || k.M != M || k.N != N || k.K != K) k = Kept{M, N, K, key, choosePlan(M, N, K, sms, pairs, bMn, epilogue)};
  return k.p;
}

ncclResult_t gemmTileLaunch(const GemmTilePlan& p, const void* A, const void* B, void* C, int M, int N, int K, cudaStream_t stream,
                            int aMn, int bMn, uint32_t* errDev, uint32_t* errHost) {
  CUtensorMap ma, mb, mc;
  DFCHECK(gemmMakeMap3(&ma, A, (uint64_t)M, (uint64_t)K, aMn, TM, BK));
  DFCHECK(gemmMakeMap3(&mb, B, (uint64_t)N, (uint64_t)K, bMn, bRows(p.pair, p.tn), BK));
  mc = ma;
  if (boxed(p.tn) && p.split == 1) DFCHECK(gemmMakeMap(&mc, C, (uint64_t)M, (uint64_t)N, 32, 32));
  CUDACHECK(oncePerDevice([] {
    cudaError_t r = cudaSuccess;
    for (const Form& f : FORMS) if (r == cudaSuccess) r = allowSharedMemory(kernelOf(f.pair, f.tn), SMEM_LIMIT);
    return r == cudaSuccess ? allowSharedMemory(kernelOf(true, 256), SMEM_LIMIT) : r;
  }));
  TileArgs g;
  memset(&g, 0, sizeof(g));
  g.C = (__nv_bfloat16*)C; g.M = M; g.N = N; g.K = K; g.aMn = aMn ? 1 : 0; g.bMn = bMn ? 1 : 0;
  g.split = p.split; g.stages = stagesOf(p.pair, p.tn, p.split, K / 64);
  g.err = errDev; g.errHost = errHost;
  const int rows = p.pair ? 2 * TM : TM, clusterSize = (p.pair ? 2 : 1) * p.split;
  const int tiles = (M + rows - 1) / rows * (N / p.tn);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(tiles * clusterSize); cfg.blockDim = dim3(NUM_THREADS); cfg.stream = stream;
  // at least the SM's shared memory times the share of its tensor memory (TN of 512 columns): CTAs that are resident
  // together, of one launch, of the next one or of another stream, then never wait for tensor memory
  cfg.dynamicSmemBytes = std::max(std::max(g.stages * stageBytes(p.pair, p.tn), EPI_BYTES) + exchangeBytes(p.tn, p.split) + BAR_BYTES + ALIGN_SLACK,
                                  228 * 1024 * p.tn / 512 - 1024);
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = clusterSize; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = clusterSize > 1 ? 2 : 1;
  CUDACHECK(cudaLaunchKernelEx(&cfg, kernelOf(p.pair, p.tn), ma, mb, mc, g));
  return ncclSuccess;
}

}  // namespace dfccl
