// Structures shared by the host runtime and the daemon kernel.
//
// Everything here is plain data laid out identically on both sides.  Roles map to
// the reference as follows (reference paths are relative to its src/):
//   Sqe / host SQ ring      - include/collectives_ofccl.h:129-145 (SQE, SQ)
//   CQ entry encoding       - include/collectives_ofccl.h:11-19,152-157
//   CollStatic              - StaticCollCtx   include/collectives_ofccl.h:320-343
//   CollDyn                 - DynamicCollCtx  include/collectives_ofccl.h:344-355
//   BlockSaved / BlockShared- BlkStatus       include/collectives_ofccl.h:171-318
// The differences are deliberate: queues have a device-resident mirror so that
// only one warp polls host memory; a collective owns flag words in
// every member's symmetric heap instead of a private communicator with FIFOs;
// the saved cursor of a parked collective is (phase, cursor) because the data
// movement between two waits never blocks.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>
#include "dfccl.h"

#define DF_MAX_RANKS 64        // ranks of one communicator the direct-access engine serves (one NVLink domain: 8 per node, up to 72 in a rack)
#define DF_MAX_BLOCKS 64       // daemon thread blocks per rank
#define DF_MAX_COLLS 2048      // collective ids per rank context (reference MAX_LENGTH = 2000)
#define DF_WARP 32

namespace dfccl {

// ---- submission queue entry: four 64-bit words, each with a 7-bit tag in its top bits that changes with every turn of
// the ring.  A word is read and written as a whole, so a reader that finds the expected tag in all four words has the
// entry, in whatever order they arrived: one look at a slot both finds and fetches an entry, and no tail word, fence or
// second round trip stands between the two.
enum SqeFlags : uint32_t {
  SQE_QUIT = 1u,          // final quit: every block saves nothing and leaves for good
  SQE_TRIGGERED = 2u,     // do not start before trigger[collId] >= trigger value (stream-ordered submit)
  SQE_SEND_STAGED = 4u,   // sendbuff is outside the symmetric heap: copy it into the staging area first
  SQE_RECV_STAGED = 8u,   // recvbuff is outside the heap: peers write staging, copy out at the end
  SQE_NEW_STATIC = 16u,   // the host has changed the collective's CollStatic (new staging areas): a copy kept by a block is stale
};
struct Sqe {
  int32_t collId;
  uint32_t flags;
  uint64_t send;          // heap offset, or raw local address when SQE_SEND_STAGED (57 bits)
  uint64_t recv;          // heap offset, or raw local address when SQE_RECV_STAGED (57 bits)
  uint32_t trigger;       // value the low half of trigger[collId] must reach (SQE_TRIGGERED)
  uint32_t epoch;         // number of this submission of the collective, counted by the host from 1: not every submission
                          // of an id has to pass through the daemon
};
struct alignas(32) SqSlot { uint64_t w[4]; };
#define DF_SQ_PAYLOAD ((1ull << 57) - 1)
// Tag of ring position `index`: 1..127, so that a slot never written to (all zero) matches nothing; the slot's previous
// contents are exactly one turn old.
static __host__ __device__ inline int log2Of(uint32_t powerOfTwo) {
#if defined(__CUDA_ARCH__)
  return 31 - __clz((int)powerOfTwo);
#else
  return __builtin_ctz(powerOfTwo);
#endif
}
static __host__ __device__ inline uint64_t sqTag(uint64_t index, uint32_t cap) { return (uint32_t)(index >> log2Of(cap)) % 127u + 1u; }
static __host__ __device__ inline SqSlot sqEncode(const Sqe& q, uint64_t tag) {
  SqSlot s;
  s.w[0] = tag << 57 | (uint64_t)(q.flags & 0x1ffu) << 48 | (uint64_t)(q.collId & 0xffff) << 32 | q.epoch;
  s.w[1] = tag << 57 | (q.send & DF_SQ_PAYLOAD);
  s.w[2] = tag << 57 | (q.recv & DF_SQ_PAYLOAD);
  s.w[3] = tag << 57 | q.trigger;
  return s;
}
static __host__ __device__ inline Sqe sqDecode(const SqSlot& s) {
  Sqe q;
  q.epoch = (uint32_t)s.w[0]; q.collId = (int16_t)(uint16_t)(s.w[0] >> 32); q.flags = (uint32_t)(s.w[0] >> 48) & 0x1ffu;
  q.send = s.w[1] & DF_SQ_PAYLOAD; q.recv = s.w[2] & DF_SQ_PAYLOAD; q.trigger = (uint32_t)s.w[3];
  return q;
}

// ---- completion entry: one 64-bit word, gen makes a slot self-validating
//   [63:32] generation of the ring slot (index / capacity + 1)   [31:24] status   [23:0] collId
static __host__ __device__ inline uint64_t cqeEncode(uint32_t gen, uint32_t status, uint32_t collId) {
  return ((uint64_t)gen << 32) | ((uint64_t)(status & 0xff) << 24) | (collId & 0xffffff);
}
static __host__ __device__ inline uint32_t cqeGen(uint64_t e) { return (uint32_t)(e >> 32); }
static __host__ __device__ inline uint32_t cqeStatus(uint64_t e) { return (uint32_t)(e >> 24) & 0xff; }
static __host__ __device__ inline uint32_t cqeColl(uint64_t e) { return (uint32_t)e & 0xffffff; }

// ---- per (collective, block, source rank) flag words, written by the source rank
struct alignas(32) FlagSlot {
  uint64_t arrive;        // epoch of the submission whose offsets are valid
  uint64_t sendOff;       // source rank's send buffer, offset in its heap; in the engine's slots under the epoch's tag (offTagged)
  uint64_t recvOff;       // source rank's recv buffer, offset in its heap, likewise
  uint64_t done;          // epoch whose data movement the source rank finished
};

// ---- phases of a collective on one block (the saved cursor)
// An offset carries the low 16 bits of its epoch: whoever finds the tag in the slot of a registered collective has the offset
// of that submission (what stood there before is exactly one epoch old), in whatever order the words of a slot arrive, so that
// posting them takes no release among ranks of one device.
#define DF_OFF_BITS 48
static __host__ __device__ inline uint64_t offTagged(uint64_t off, uint32_t epoch) { return (off & ((1ull << DF_OFF_BITS) - 1)) | (uint64_t)(epoch & 0xffffu) << DF_OFF_BITS; }
static __host__ __device__ inline bool offCurrent(uint64_t w, uint32_t epoch) { return (uint32_t)(w >> DF_OFF_BITS) == (epoch & 0xffffu); }
static __host__ __device__ inline uint64_t offValue(uint64_t w) { return w & ((1ull << DF_OFF_BITS) - 1); }

enum Phase : int32_t {
  PH_TRIGGER = 0,         // bounded wait: local trigger word
  PH_COPY_IN = 1,         // local copy user send buffer -> staging (unregistered buffers)
  PH_POST_ARRIVE = 2,     // write my offsets + epoch into every peer's flag slot
  PH_WAIT_ARRIVE = 3,     // bounded wait: all peers arrived
  PH_DATA = 4,            // move data; never blocks
  PH_POST_DONE = 5,       // fence, then write done = epoch into every peer's flag slot
  PH_WAIT_DONE = 6,       // bounded wait: all peers done
  PH_COPY_OUT = 7,        // local copy staging -> user recv buffer
  PH_COMPLETE = 8,
};

enum CollStatus : uint32_t { ST_OK = 0, ST_TIMEOUT = 1, ST_ABORTED = 2, ST_BAD_ARG = 3 };
// The word in which the blocks of a collective count themselves and leave their verdicts: [7:0] how many are done, and of those
// [15:8] how many timed out, [23:16] were aborted, [31:24] met a bad argument (DF_MAX_BLOCKS of each at most).
static __host__ __device__ inline uint32_t doneWord(uint32_t status) { return 1u | (status != ST_OK ? 1u << (8u * (status <= ST_BAD_ARG ? status : ST_TIMEOUT)) : 0u); }
// The collective's status where the causes differ: one that a block has reported.  (A wait that ran out is the cause of an
// abort that follows it.)
static __host__ __device__ inline uint32_t doneVerdict(uint32_t w) { return w >> 24 ? ST_BAD_ARG : w >> 8 & 0xffu ? ST_TIMEOUT : w >> 16 & 0xffu ? ST_ABORTED : ST_OK; }

// ---- immutable description of a registered collective (one per collId per rank)
struct alignas(16) CollStatic {
  int32_t kind;           // dfcclColl_t
  int32_t inType, outType;
  int32_t op;             // ncclSum..ncclMin (Avg is folded into scale / postDiv at prepare time)
  int32_t nranks, rank, root;
  int32_t nBlocks;        // blocks that take part; the block at relative index b handles slice b of the data
  int32_t algo;           // dfcclAlgo_t actually used
  int32_t postDiv;        // integer average: divide the sum by this (0 = off)
  int32_t valid;
  int32_t blockBase;      // daemon block that plays relative block 0 of this collective: the nBlocks participants are
                          // blockBase, blockBase + 1, ... (mod the daemon's block count), so that collectives too small
                          // for every block do not all land on the first blocks.  A per-rank choice: ranks meet by
                          // relative index only.
  int32_t oneDevice;      // all members are ranks on this GPU, their heaps in its memory: what orders one member's
                          // accesses for another is a fence of GPU scope (0.24 - 0.45 us against 1.4 - 1.8 us)
  int32_t esIn, esOut;    // bytes of an element
  int32_t reduces;        // the unit of the partition below: elements (reducing kinds) or bytes (copying kinds)
  // partition, so that no block divides (planColl): block b moves units [per b, per (b + 1)) of `total`, and of such a range
  // member r owns [perShard r, perShard (r + 1)) in the two-shot schedules; the one range that is neither whole nor empty
  // is cut at multiples of perShardLast
  uint64_t total, per, perShard, perShardLast;
  uint64_t sliceUnits;    // a visit moves at most this many (0: no limit)
  double scale;           // multiplies the reduced value (1.0 = off)
  uint64_t count;         // elements, NCCL convention of the kind
  uint64_t stagingSendOff, stagingRecvOff;      // my heap offsets of staging areas (0 = none)
  FlagSlot* myFlags;                            // [nBlocks][nranks] in my heap
  FlagSlot* peerFlags[DF_MAX_RANKS];            // the same block of member j, as mapped here
  char* peerHeap[DF_MAX_RANKS];                 // heap base of member j, as mapped here
  // NVLS schedule: the arena's multicast mapping (null where the view is emulated), the members' arena
  // blocks for the emulation (host backend; null on GPUs), and this collective's staging slots in the arena
  char* mcHeap;
  char** nvlsPeers;
  uint64_t nvlsIn, nvlsOut;
  // push schedule: slot area of member j as mapped here, laid out [2 parities][nranks writers][pushSlotBytes]
  char* peerPush[DF_MAX_RANKS];
  uint64_t pushSlotBytes;
};

// Fills the fields above from kind, types, count, nranks and nBlocks; sliceBytes as in RankConst.
inline void planColl(CollStatic* c, uint64_t sliceBytes) {
  auto size = [](int t) { return t == ncclInt8 || t == ncclUint8 ? 1 : t == ncclFloat16 || t == ncclBfloat16 ? 2 : t == ncclInt32 || t == ncclUint32 || t == ncclFloat32 ? 4 : 8; };
  c->esIn = size(c->inType); c->esOut = size(c->outType);
  c->reduces = c->kind == dfcclCollAllReduce || c->kind == dfcclCollReduce || c->kind == dfcclCollReduceScatter;
  c->total = c->reduces ? c->count : c->count * (uint64_t)c->esIn;
  auto cut = [](uint64_t total, int parts) { return ((total + parts - 1) / parts + 15) & ~(uint64_t)15; };
  c->per = cut(c->total, c->nBlocks);
  c->perShard = cut(c->per, c->nranks);
  c->perShardLast = c->per ? cut(c->total % c->per, c->nranks) : 0;
  const uint64_t unit = c->reduces ? (uint64_t)c->esIn : 1, slice = sliceBytes / unit & ~(uint64_t)15;
  c->sliceUnits = sliceBytes == 0 ? 0 : slice < 16 ? 16 : slice;
}

#define DF_META_VALID (1u << 16)
inline uint32_t collMeta(const CollStatic& c) { return c.valid ? DF_META_VALID | (uint32_t)c.nBlocks | (uint32_t)c.blockBase << 8 : 0u; }

// ---- mutable per (block, collective) state; what a context switch saves and loads
struct alignas(16) CollDyn {
  uint64_t send, recv;    // this submission's buffers (offset or raw address, see Sqe)
  uint64_t trigger;       // low 32 bits count
  uint64_t cursor;        // progress inside PH_DATA / copies when sliced
  uint32_t epoch;         // number of the running submission (0 = none yet)
  int32_t phase;
  uint32_t sqeFlags;
  uint32_t status;
  uint64_t stallSinceNs;  // first unsuccessful poll of the current wait (0 = not stalled)
  uint32_t patience;      // polls a wait of this submission may spend at least: raised after every wait that succeeded
                          // (reference: RECV_SUCCESS_FACTOR, src/collectives_ofccl/device/ofccl_prims_simple.h:79-88)
  uint32_t pad;
};

// ---- host-pinned control words
struct DaemonCtl {
  volatile uint32_t abortFlag;     // host sets; every block leaves at its next poll
  volatile uint32_t alive;         // host sets at launch; last exiting block clears
  volatile uint32_t finalQuit;     // device sets when it consumed the quit entry
  volatile uint32_t pad;           // stream-ordered kernels store a non-zero CollStatus here on failure
  volatile uint64_t launches;
  volatile uint64_t voluntaryQuits;
  // host sets while a stream is (or will be) parked on a completion word of this context: the running
  // instance then stays resident instead of leaving when it is idle or stalled, so that no relaunch
  // from a host thread is needed at the moment the GPU waits; cleared when nothing is outstanding
  volatile uint32_t hold;
  volatile uint32_t pad1;
};

struct DevStats {                  // per block, device memory
  unsigned long long ctxSwitches, ctxSaves, ctxLoads, waitPolls, waitTimeouts, bytesReduced, bytesCopied,
      maxSwitchNs, totalSwitchNs, sqesSeen, collsDone, visits,
      yields,        // data phases left at a slice boundary because other work was queued
      passes,        // scheduler passes (trigger poll + task-queue walk + queue maintenance)
      nsTriggers, nsWalk, nsQueues;   // where thread 0 saw the passes' time go: trigger list, task-queue walk, queue upkeep
};

struct TraceEvent { uint64_t ns; uint16_t block; uint16_t event; int32_t collId; };
enum TraceKind : uint16_t { TR_SQE = 1,          // submission consumed by this block
                            TR_START = 2,        // released by its stream (or submitted from the host)
                            TR_STALL = 3,        // a wait ran out of budget: the collective stays queued, the block moves on
                            TR_ARRIVED = 4,      // every peer has arrived
                            TR_DATA_BEGIN = 5, TR_DATA_END = 6,
                            TR_DONE = 7,         // this block's part is complete (the last block publishes the completion)
                            TR_QUIT = 8, TR_LAUNCH = 9,
                            TR_PEERS_DONE = 10,  // every peer has finished its data movement
                            TR_YIELD = 11 };     // data phase left at a slice boundary

#define DF_MAX_ACTIVE 2048   // task-queue capacity per block (>= DF_MAX_COLLS: one outstanding submit per id)

struct BlockSaved {                // survives a voluntary quit (reference: DynamicBlkStatus + activeCollIds)
  uint64_t frontier;               // SQ entries consumed by this block
  uint32_t nActive;
  uint32_t exited;
  uint32_t nTrig;                  // stream-ordered submissions whose stream has not released them yet
  uint32_t pad;
  uint16_t active[DF_MAX_ACTIVE];
  uint16_t trigColl[DF_MAX_ACTIVE];
  uint32_t trigVal[DF_MAX_ACTIVE];
};

// ---- everything the daemon needs for one rank; lives in device memory (host memory for the host backend)
// What does not change after finalize: every block keeps a copy (BlockShared::k).
struct RankConst {
  // Submission path: the host writes entries into a ring in pinned memory with plain stores; ONE warp per rank (the
  // service warp of block 0) polls it and copies new entries into the ring in device memory that the blocks poll.
  // (A load of pinned host memory is a PCIe round trip, and such loads from many blocks queue behind one another; a
  // write by the host through stream memory operations costs it a driver call and the device a fence per word.)
  const volatile SqSlot* hostSq;   // null: the host writes devSq itself (host backend)
  volatile SqSlot* devSq;
  uint32_t sqCap;                  // power of two
  uint32_t pad0;
  volatile uint64_t* hostFrontier; // pinned, [nBlocks]: entries consumed by each block (posted stores; flow control for the host)
  volatile uint32_t* abortWord;    // where this rank's abort request is polled: device memory for the daemon (the host
                                   // writes it with a stream memory operation), the pinned control block otherwise
  // completion path
  volatile uint64_t* hostCq;       // pinned ring read by the poller
  uint32_t cqCap;                  // power of two
  uint32_t nBlocks;
  // tables
  CollStatic* colls;               // [maxColls]
  uint32_t* meta;                  // [maxColls] what a block needs to know to take or skip an entry: nBlocks | blockBase << 8 |
                                   // DF_META_VALID; never written after finalize
  CollDyn* dyn;                    // [nBlocks][maxColls]
  uint32_t* doneCount;             // [maxColls] blocks that finished the current submission and their verdicts (doneWord; a collective
                                   // that runs in its stream counts its kernel's blocks here)
  volatile uint64_t* doneEpoch;    // [maxColls] device flag: epoch of the last finished submission
  volatile uint64_t* trigger;      // [maxColls] device flag written by stream memory operations
  BlockSaved* saved;               // [nBlocks]
  DevStats* stats;                 // [nBlocks]
  TraceEvent* trace;               // ring, or null
  uint32_t traceCap;
  uint32_t maxColls;
  DaemonCtl* ctl;                  // pinned
  // tunables (reference: src/enqueue_ofccl.cc:1287-1297)
  uint32_t spinBudget;             // BASE_CTX_SWITCH_THRESHOLD
  uint32_t headTries;              // NUM_TRY_TASKQ_HEAD
  uint32_t recvSuccessFactor;      // RECV_SUCCESS_FACTOR
  uint64_t idleQuitNs;             // leave after this long with an empty task queue and no new entry
  uint64_t stallQuitNs;            // leave after this long with only stalled collectives
  uint64_t trigQuitNs;             // leave after this long with nothing but submissions that wait for their stream
  uint64_t waitTimeoutNs;          // a single wait older than this fails with ST_TIMEOUT (0 = never)
  uint64_t maxLifetimeNs;          // one launch of the daemon leaves after this long regardless of its state (0 = never)
  uint64_t sliceBytes;             // PH_DATA yields after this many bytes when others are queued (0 = never)
};
// Polls of a wait beside submissions that a stream has not released yet: their trigger words are looked at in between.
static __host__ __device__ inline uint32_t pollsBesideTriggers(const RankConst* k) { return (k->spinBudget + 7u) / 8u * k->headTries; }
struct RankDev : RankConst {
  uint64_t svcHead;                // entries the service warp has copied
  uint64_t devCqTail;
  uint64_t traceHead;
  uint32_t exitedBlocks;
  volatile uint32_t quitting;      // a block left voluntarily during this launch
  uint32_t saEpoch;                // stream-ordered kernels: number of collectives this communicator has finished (their epoch
                                   // lives on the device so that a captured launch finds the right one at every replay)
};

}  // namespace dfccl
