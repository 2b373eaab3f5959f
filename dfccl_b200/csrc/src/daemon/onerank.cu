// Collectives of a one-rank communicator.  Every kind is the same thing there: out = cast(scale x in) over the call's
// elements, or a copy.  Nobody has to be waited for, so the work needs no flags, no staging of buffers outside the
// symmetric heap and no limit on the blocks: it is one streaming kernel over the whole GPU.
//
// Bound: HBM (or L2 for what fits there).  A block of 256 threads takes 1024 consecutive 16-byte packs, four per
// thread and all four loads before the first store, so that 5 resident blocks (48 registers a thread) keep 80 KB per SM in
// flight; calls too small to give every SM such a block take one pack per thread instead (more blocks, shorter chains).
// The blocks come up while the kernel in front of them in the stream drains.  bf16 -> fp32 packs are stored as whole 32-byte sectors.
// Measured: all-reduce of 8388611 fp32 values in ordinary tensors 11.4 us = 5.9 TB/s read + write (13.9 without early blocks; the
// collective kernel, which stages such buffers into the heap and out again on 64 blocks, 64.7).
#include "../device/engine.h"
#include "../device/launch.h"
#include "../gemm/tc_common.h"
#include "../common/log.h"
#include <algorithm>

namespace dfccl {
namespace {

constexpr int THREADS = 256;
constexpr int CLUSTER = 8;                 // blocks of a short registered collective: one cluster

struct OneRankArgs {
  const char* src;
  char* dst;
  uint64_t n;                // elements (bytes for a plain copy)
  uint64_t head;             // elements in front of the first pack (brings both pointers to the 16-byte grid)
  uint64_t nPacks;           // packs of 16 source bytes
  double scale;
  int postDiv;
  OneRankDone done;          // registered collective: where the completion goes (rd null: a stream-ordered call, nowhere)
};

// One element of the head, the ragged tail, or of buffers that do not line up.
template <typename Tin, typename Tout>
__device__ __forceinline__ void oneElem(const OneRankArgs& a, uint64_t e) {
  typedef typename Elem<Tin>::Acc A;
  Tin v = *((const Tin*)a.src + e);
  A acc = Elem<Tin>::up(v);
  *((Tout*)a.dst + e) = Elem<Tout>::down(finish<Tin, Tout>(acc, a.scale, a.postDiv));
}

// The place of the host's entry in its ring.
__device__ __forceinline__ unsigned long long takePlace(const OneRankDone& done) { return atomic_add_u64((unsigned long long*)&done.rd->devCqTail, 1ull); }
__device__ __forceinline__ void publishDone(const OneRankDone& done, unsigned long long idx) {
  RankDev* rd = done.rd;
  fence_acq_rel_sys();
  st_relaxed_sys_u64(&rd->doneEpoch[done.coll], ((uint64_t)ST_OK << 56) | done.epoch);
  st_relaxed_sys_u64(&rd->hostCq[idx & (rd->cqCap - 1)], cqeEncode((uint32_t)(idx / rd->cqCap) + 1u, ST_OK, (uint32_t)done.coll));
}

// SHORT: the whole call is one cluster of blocks, which meet at the cluster's barrier before one thread publishes, instead of
// counting themselves in global memory (a fence and an atomic, two round trips to L2 at the end of a kernel that moves 64 KB).  Up
// to what a cluster holds with four packs a thread in flight; eight calls behind one another in a stream, blocks that count
// themselves / one cluster, us: 8 KB 38.8 / 35.5, 64 KB 45.8 / 36.3, 128 KB (the limit) 47.4 / 37.2.
// What is left of such a call (4.5 us): 1.35 until the kernel in front is known to have ended, 0.6 for the data, 0.65 for the cluster's
// barrier, 1.9 for the system-wide fence and the entry, whose place was asked for in front of the loads (eight of
// 64 KB 36.1 -> 35.5, of 128 KB as fp32 40.1 -> 38.5, of 16 KB and less the same).
// The blocks may come up while the kernel in front of them in the stream still runs, and wait for its end before they read.
template <typename Tin, typename Tout, bool COPY, int U, bool SHORT>
__global__ void __launch_bounds__(THREADS) dfcclOneRankKernel(const OneRankArgs a) {
  typedef typename Elem<Tin>::Acc A;
  constexpr int V = 16 / (int)sizeof(Tin);
  constexpr int OUTB = V * (int)sizeof(Tout);
  constexpr int NW = (OUTB + 15) / 16;
  // (a cluster shares out every THREADS packs, so that all of its SMs load)
  constexpr int STEP = SHORT ? CLUSTER * THREADS : THREADS;
  const uint64_t p0 = (uint64_t)blockIdx.x * (SHORT ? THREADS : THREADS * U) + threadIdx.x;
  const uint4* s = (const uint4*)(a.src + a.head * sizeof(Tin));
  char* d = a.dst + a.head * sizeof(Tout);
  tc::grid_dependency_wait();
  tc::grid_launch_dependents();
  // (a place taken now keeps the places behind it waiting until this call is done: a matter of microseconds where it is SHORT)
  unsigned long long place = 0;
  if (SHORT && blockIdx.x == 0 && threadIdx.x == 0) place = takePlace(a.done);
  uint4 v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) if (p0 + u * STEP < a.nPacks) v[u] = s[p0 + u * STEP];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (p0 + u * STEP >= a.nPacks) continue;
    char* o = d + (p0 + u * STEP) * OUTB;
    if (COPY) { *(uint4*)o = v[u]; continue; }
    A r[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      r[k] = (A)Lane<Tin>::get(v[u], k);
      if (Elem<Tin>::isFloat) r[k] = r[k] * (A)a.scale;                    // (times one changes nothing)
      else if (a.postDiv) r[k] = r[k] / (A)a.postDiv;
      else if (a.scale != 1.0) r[k] = (A)((double)r[k] * a.scale);
    }
    uint4 ow[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) ow[w] = make_uint4(0u, 0u, 0u, 0u);
    packAll<Tout, A, V>(ow, r);
    if (OUTB == 8) *(uint2*)o = make_uint2(ow[0].x, ow[0].y);
    else if (OUTB == 32) st32(o, ow[0], ow[NW - 1], ((uintptr_t)o & 31) == 0);
    else {
#pragma unroll
      for (int w = 0; w < OUTB / 16; ++w) ((uint4*)o)[w] = ow[w];
    }
  }
  // what is not in a pack
  const uint64_t tail0 = a.head + a.nPacks * V, rest = a.head + (a.n - tail0);
  for (uint64_t i = (uint64_t)blockIdx.x * THREADS + threadIdx.x; i < rest; i += (uint64_t)gridDim.x * THREADS) {
    const uint64_t e = i < a.head ? i : tail0 + (i - a.head);
    if (COPY) a.dst[e] = a.src[e]; else oneElem<Tin, Tout>(a, e);
  }
  if (SHORT) {
    tc::cluster_sync_all();
    if (blockIdx.x == 0 && threadIdx.x == 0) publishDone(a.done, place);
    return;
  }
  if (a.done.rd == nullptr) return;
  // The last block out publishes the completion, as the daemon's blocks do, but with one system-wide fence for the device
  // flag and the host's entry together, and with the entry's index on its way before it: every step here is a round trip
  // to L2 at the end of a kernel that may have moved 64 KB (6.3 us, of which the data takes 2).
  __syncthreads();
  if (threadIdx.x == 0) {
    RankDev* rd = a.done.rd;
    if (gridDim.x > 1) {
      fence_gpu();
      uint32_t* count = &rd->doneCount[a.done.coll];
      if (atomic_add_u32(count, 1u) + 1u != gridDim.x) return;
      *(volatile uint32_t*)count = 0u;
    }
    publishDone(a.done, takePlace(a.done));
  }
}

// With tracing on: in the stream before and after the data kernel, which then publishes nothing itself (events written there
// cost it 0.1 - 0.3 us with tracing off, 33 MB in 13.65 us instead of 13.38).
__global__ void dfcclOneRankTraceKernel(const OneRankDone done, bool end) {
  if (!end) {
    trace(done.rd, 0, TR_SQE, done.coll);
    trace(done.rd, 0, TR_START, done.coll);
    trace(done.rd, 0, TR_DATA_BEGIN, done.coll);
    return;
  }
  trace(done.rd, 0, TR_DATA_END, done.coll);
  trace(done.rd, 0, TR_DONE, done.coll);
  publishDone(done, takePlace(done));
}

template <typename Tin, typename Tout, bool COPY>
ncclResult_t launchTyped(OneRankArgs a, int sms, cudaStream_t stream) {
  constexpr int V = 16 / (int)sizeof(Tin);
  constexpr int DA = V * (int)sizeof(Tout) >= 16 ? 16 : V * (int)sizeof(Tout);       // alignment the vector stores need
  // `head` elements bring the destination to its alignment; the packs are used when the source is aligned there too
  const uint64_t dphase = (uintptr_t)a.dst & (DA - 1);
  bool vec = dphase % sizeof(Tout) == 0;
  uint64_t head = vec ? ((DA - dphase) % DA) / sizeof(Tout) : 0;
  if (head > a.n) head = a.n;
  vec = vec && ((uintptr_t)(a.src + head * sizeof(Tin)) & 15) == 0;
  a.head = vec ? head : 0;
  a.nPacks = vec ? (a.n - head) / V : 0;
  const uint64_t loose = a.n - a.nPacks * V;
  const uint64_t looseBlocks = std::min<uint64_t>((loose + THREADS - 1) / THREADS, (uint64_t)sms * 8);
  void (*kernel)(const OneRankArgs) = dfcclOneRankKernel<Tin, Tout, COPY, 1, false>;
  uint64_t grid = std::max<uint64_t>(1, std::max((a.nPacks + THREADS - 1) / THREADS, looseBlocks));
  int cluster = 1;
  if (a.done.rd && a.nPacks <= CLUSTER * THREADS * 4 && looseBlocks <= CLUSTER) {
    kernel = dfcclOneRankKernel<Tin, Tout, COPY, 4, true>;
    grid = cluster = CLUSTER;
  } else if (a.nPacks >= (uint64_t)sms * THREADS * 4) {
    kernel = dfcclOneRankKernel<Tin, Tout, COPY, 4, false>;
    grid = std::max((a.nPacks + THREADS * 4 - 1) / (THREADS * 4), looseBlocks);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3(THREADS); cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = cluster > 1 ? 2 : 1;
  CUDACHECK(cudaLaunchKernelEx(&cfg, kernel, a));
  return ncclSuccess;
}

int smCount() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

ncclResult_t launchOneRankCuda(const CollStatic& cs, const void* send, void* recv, cudaStream_t stream, const OneRankDone* done, bool traced) {
  if (done && traced) {
    dfcclOneRankTraceKernel<<<1, 1, 0, stream>>>(*done, false);
    CUDACHECK(cudaGetLastError());
    DFCHECK(launchOneRankCuda(cs, send, recv, stream, nullptr, false));
    dfcclOneRankTraceKernel<<<1, 1, 0, stream>>>(*done, true);
    CUDACHECK(cudaGetLastError());
    return ncclSuccess;
  }
  OneRankArgs a;
  memset(&a, 0, sizeof(a));
  if (done) a.done = *done;
  a.src = (const char*)send; a.dst = (char*)recv; a.n = cs.count; a.scale = cs.scale; a.postDiv = cs.postDiv;
  const bool reduces = cs.kind == dfcclCollAllReduce || cs.kind == dfcclCollReduce || cs.kind == dfcclCollReduceScatter;
  const bool plain = cs.inType == cs.outType && (!reduces || (cs.scale == 1.0 && cs.postDiv <= 1));
  const int sms = smCount();
  if (plain) {
    a.n = cs.count * (uint64_t)dtypeSize(cs.inType);
    if (send == recv) {                                  // in place: already where it belongs
      if (!done) return ncclSuccess;
      a.n = 0;
    }
    return launchTyped<uint8_t, uint8_t, true>(a, sms, stream);
  }
  if (cs.inType == cs.outType) {
    switch (cs.inType) {
#ifndef DF_FAST_BUILD
      case ncclInt8: return launchTyped<int8_t, int8_t, false>(a, sms, stream);
      case ncclUint8: return launchTyped<uint8_t, uint8_t, false>(a, sms, stream);
      case ncclInt32: return launchTyped<int32_t, int32_t, false>(a, sms, stream);
      case ncclUint32: return launchTyped<uint32_t, uint32_t, false>(a, sms, stream);
      case ncclInt64: return launchTyped<int64_t, int64_t, false>(a, sms, stream);
      case ncclUint64: return launchTyped<uint64_t, uint64_t, false>(a, sms, stream);
      case ncclFloat16: return launchTyped<__half, __half, false>(a, sms, stream);
      case ncclFloat64: return launchTyped<double, double, false>(a, sms, stream);
#endif
      case ncclFloat32: return launchTyped<float, float, false>(a, sms, stream);
      case ncclBfloat16: return launchTyped<__nv_bfloat16, __nv_bfloat16, false>(a, sms, stream);
      default: return ncclInvalidArgument;
    }
  }
  if (cs.inType == ncclBfloat16 && cs.outType == ncclFloat32) return launchTyped<__nv_bfloat16, float, false>(a, sms, stream);
  if (cs.inType == ncclFloat16 && cs.outType == ncclFloat32) return launchTyped<__half, float, false>(a, sms, stream);
  if (cs.inType == ncclFloat32 && cs.outType == ncclBfloat16) return launchTyped<float, __nv_bfloat16, false>(a, sms, stream);
  if (cs.inType == ncclFloat32 && cs.outType == ncclFloat16) return launchTyped<float, __half, false>(a, sms, stream);
  return ncclInvalidArgument;
}

}  // namespace dfccl
