// Host-callable launchers of the device runtime (CUDA) and of its host-thread twin.
#pragma once
#include "types.h"
#include "dfccl.h"

namespace dfccl {

// Persistent daemon for `nRanks` rank contexts that share one device: one launch,
// grid = nRanks * blocksPerRank.  With more than one rank the launch is cooperative,
// so that all blocks are co-resident (blocks of different ranks wait on one another).
ncclResult_t launchDaemonCuda(RankDev** devRankTable, int nRanks, int blocksPerRank, int threads, cudaStream_t stream);

// One collective as a plain kernel on the caller's stream (stream-ordered nccl* interface).
ncclResult_t launchStandaloneCuda(RankDev* rd, const CollStatic& cs, uint64_t send, uint64_t recv, uint32_t epoch,
                                  uint32_t sqeFlags, int threads, cudaStream_t stream);

// The same on a one-rank communicator: one streaming kernel, buffers used where they are.  With `done` the kernel also
// publishes the completion of a registered collective (device flag and completion entry); `traced`: and the daemon's events
// for it, as block 0's.
struct OneRankDone { RankDev* rd; int32_t coll; uint32_t epoch; };
ncclResult_t launchOneRankCuda(const CollStatic& cs, const void* send, void* recv, cudaStream_t stream, const OneRankDone* done = nullptr,
                               bool traced = false);

// Force the lazily loaded kernels of the runtime into the context (no launch).
ncclResult_t warmRuntimeKernels();

// Largest grid of the daemon kernel that is guaranteed co-resident on `device`.
ncclResult_t daemonMaxResidentBlocks(int device, int threads, int* blocks);

// Host backend: the same code with one OS thread per block.  Both calls block until
// every "block" has returned.
void runDaemonHost(RankDev** rankTable, int nRanks, int blocksPerRank);
void runStandaloneHost(RankDev* rd, const CollStatic& cs, uint64_t send, uint64_t recv, uint32_t epoch, uint32_t sqeFlags);

}  // namespace dfccl
