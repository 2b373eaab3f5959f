// Step engine: one registered collective, executed by one block, as a resumable
// sequence of phases (types.h: Phase).  Two kinds of phases exist:
//   * bounded waits (PH_TRIGGER, PH_WAIT_ARRIVE, PH_WAIT_DONE) poll words in LOCAL
//     memory that a peer, the host or a stream memory operation writes.  A wait
//     that runs out of budget returns to the scheduler without side effects: it
//     consumed nothing and wrote nothing, so parking the collective is saving
//     (phase, cursor) - there is no connection state to unwind.
//   * actions (posting flags, moving data) never wait for anybody.
// This replaces the reference's preemptible ring primitives, where a context
// switch had to unwind a half-executed slice and re-synchronise every thread role
// (src/collectives_ofccl/device/ofccl_prims_simple.h:118-140,217-491 and the
// resumable ring loops in ofccl_all_reduce.h:44-217): on an NVSwitch fabric every
// peer is one hop away, so each collective is "everybody arrived -> direct loads
// and stores of peer buffers -> everybody done" and the only blocking points are
// the two rendezvous.
//
// Schedules (kind x algo), all expressed as N-source / M-destination reduce-copy
// (plus the push schedule of small all-reduces: inputs are written into slots at the peers together with the arrival
// flag, every rank reduces locally and is done - one NVLink hop, no staging, no done handshake):
//   AllReduce two-shot  : block b, rank r owns shard r of slice b: reads it from all
//                         ranks, reduces, scales, casts, writes it to all ranks.
//   AllReduce one-shot  : every rank reads slice b from all ranks, writes only itself.
//   AllGather           : rank r pushes its slice b into every rank's output.
//   ReduceScatter       : rank r reads slice b of chunk r from all ranks.
//   Broadcast           : non-roots pull slice b from the root.
//   Reduce              : like two-shot AllReduce, but shards are written to the root only.
#pragma once
#include "datapath.h"
#include "nvls.h"
#include "platform.h"
#include "types.h"
namespace dfccl {

enum RunResult : int { RC_DONE = 0, RC_STALLED = 1, RC_YIELD = 2 };

struct BlockShared {
  RankConst k;                   // the rank's constants: a look at global memory is a round trip to L2 after every fence
  CollStatic cs;                 // static context of the loaded collective
  CollDyn dyn;                   // its dynamic context (authoritative copy while loaded)
  DataArgs args;
  int32_t loadedColl;            // -1 = nothing loaded
  int32_t standalone;            // 1 = stream-ordered kernel: no queues, completion is the kernel's end
  int32_t dynDirty;
  int32_t waitOk;
  uint32_t waitSpins;
  int32_t ctl0, ctl1;
  uint64_t ctl64;
  DevStats stats;
  uint64_t frontier;
  uint64_t frontierSeen;         // as last reported to the host
  uint64_t stuckAt;              // an entry that the block has met and cannot take yet (~0: none): no reason to end a wait
  uint32_t nParked;              // entries of the task queue with a wait mark, as of the end of the last pass
  uint32_t nActive;
  uint32_t quit;                 // 1 = voluntary, 2 = final, 3 = abort
  volatile uint32_t svcStop;     // the block is leaving: so does its service warp
  uint32_t abortSeen;            // the host's abort flag as last read by thread 0 (the flag lives in host memory: one
                                 // read costs a PCIe round trip, so it is sampled once per scheduler pass, not per wait)
  // peers' buffer offsets of the running submission, fetched by one lane per peer (one memory round trip for all)
  uint64_t peerSend[DF_MAX_RANKS], peerRecv[DF_MAX_RANKS];
  // stream-ordered submissions not yet released by their stream: polled all at once, one thread per entry,
  // without loading any context; a released one joins the task queue
  uint32_t nTrig;
  uint32_t trigFired;
  // what consuming an entry needs to know of its collective, so that it costs no load of the tables: RankDev::meta, and
  // whether this block still works on the previous submission
  uint32_t meta[DF_MAX_COLLS];
  uint32_t busy[DF_MAX_COLLS / 32];
  uint16_t active[DF_MAX_ACTIVE];
  // per task-queue entry: 0 = needs a visit, 1 = parked in the wait for the peers' arrival, 2 = parked in the wait for
  // their done flags.  Parked entries are not visited (a visit loads the context and polls for a while); their flag
  // words are looked at by one thread each in a scan over the whole queue, which marks the ready ones for a visit.
  uint8_t actWait[DF_MAX_ACTIVE];
  uint32_t nReady;
  uint32_t ctl1Full;               // this pass visits parked entries too (set by thread 0 at the end of the previous pass)
  uint16_t trigColl[DF_MAX_ACTIVE];
  uint32_t trigVal[DF_MAX_ACTIVE];  // low 32 bits of the value the trigger word must reach
};

static DF_HD_NOINLINE void traceEvent(RankDev* rd, int b, uint16_t ev, int coll) {
  unsigned long long i = atomic_add_u64((unsigned long long*)&rd->traceHead, 1ull);
  TraceEvent* e = &rd->trace[i & (rd->traceCap - 1)];
  e->ns = df_now_ns(); e->block = (uint16_t)b; e->event = ev; e->collId = coll;
}
DF_HD void trace(RankDev* rd, int b, uint16_t ev, int coll) { if (rd->trace != nullptr) traceEvent(rd, b, ev, coll); }
DF_HD void trace(const BlockShared* sh, RankDev* rd, int b, uint16_t ev, int coll) { if (sh->k.trace != nullptr) traceEvent(rd, b, ev, coll); }

// Entry `index` of the device ring, if it is there.
DF_HD bool sqPeek(const RankConst* rd, uint64_t index, SqSlot* out) {
  const volatile uint64_t* w = rd->devSq[index & (rd->sqCap - 1)].w;
  ld_relaxed_sys_2u64(w, &out->w[0], &out->w[1]);
  ld_relaxed_sys_2u64(w + 2, &out->w[2], &out->w[3]);
  const uint64_t tag = sqTag(index, rd->sqCap);
  return (out->w[0] >> 57) == tag && (out->w[1] >> 57) == tag && (out->w[2] >> 57) == tag && (out->w[3] >> 57) == tag;
}

// Orders this rank's accesses with those of the members it exchanges flags with.
DF_HD void fence_members(const CollStatic* c) {
  if (c->oneDevice) fence_acq_rel_gpu(); else fence_sys();
}

DF_HD uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

DF_HD bool abortRequested(const RankConst* rd) {
  return ctl_load(rd->abortWord ? rd->abortWord : &rd->ctl->abortFlag) != 0;
}

// bytes of the user's send / recv buffer (staging copies)
DF_HD uint64_t sendBytes(const CollStatic* c) {
  uint64_t e = dtypeSize(c->inType);
  switch (c->kind) {
    case dfcclCollReduceScatter: return c->count * c->nranks * e;
    default: return c->count * e;
  }
}
DF_HD uint64_t recvBytes(const CollStatic* c) {
  uint64_t e = dtypeSize(c->outType);
  switch (c->kind) {
    case dfcclCollAllGather: return c->count * c->nranks * e;
    default: return c->count * e;
  }
}

// Relative index of daemon block b in collective c (>= c->nBlocks: b takes no part).  Flags, data partitions and
// staging partitions are indexed by it; per-block state (saved contexts, statistics, trace) by the block itself.
DF_HD int relBlock(int nBlocks, const CollStatic* c, int b) {
  const int r = b - c->blockBase;
  return r < 0 ? r + nBlocks : r;
}

// ---- context switch: load / save the (static, dynamic) context of a collective
DF_HD void loadColl(BlockShared* sh, RankDev* rd, int b, int coll) {
  if (sh->loadedColl == coll) return;
  const int tid = df_tid(), nt = df_nthreads();
  df_warp_sync();                                      // (thread 0 has written the phase it left; the lanes beside it save it)
  uint64_t t0 = 0;
  if (tid == 0) t0 = df_now_ns();
  if (sh->loadedColl >= 0 && sh->dynDirty) {           // park the previous one
    CollDyn* g = &sh->k.dyn[(uint64_t)b * sh->k.maxColls + sh->loadedColl];
    const uint4* s = (const uint4*)&sh->dyn;
    for (int i = tid; i < (int)(sizeof(CollDyn) / 16); i += nt) ((uint4*)g)[i] = s[i];
    if (tid == 0) sh->stats.ctxSaves++;
  }
  df_sync();
  {
    const uint4* s = (const uint4*)&sh->k.colls[coll];
    uint4* d = (uint4*)&sh->cs;
    for (int i = tid; i < (int)(sizeof(CollStatic) / 16); i += nt) d[i] = s[i];
    const uint4* sd = (const uint4*)&sh->k.dyn[(uint64_t)b * sh->k.maxColls + coll];
    uint4* dd = (uint4*)&sh->dyn;
    for (int i = tid; i < (int)(sizeof(CollDyn) / 16); i += nt) dd[i] = sd[i];
  }
  if (tid == 0) {
    if (sh->loadedColl >= 0) {
      sh->stats.ctxSwitches++;
      uint64_t dt = df_now_ns() - t0;
      sh->stats.totalSwitchNs += dt;
      if (dt > sh->stats.maxSwitchNs) sh->stats.maxSwitchNs = dt;
    }
    sh->stats.ctxLoads++;
    sh->loadedColl = coll;
    sh->dynDirty = 0;
  }
  df_sync();
}

DF_HD void saveLoaded(BlockShared* sh, RankDev* rd, int b) {
  if (sh->loadedColl >= 0 && sh->dynDirty && df_tid() == 0) {
    rd->dyn[(uint64_t)b * rd->maxColls + sh->loadedColl] = sh->dyn;
    sh->stats.ctxSaves++;
    sh->dynDirty = 0;
  }
}

DF_HD uint64_t mySendOff(const BlockShared* sh) {
  return (sh->dyn.sqeFlags & SQE_SEND_STAGED) ? sh->cs.stagingSendOff : sh->dyn.send;
}
DF_HD uint64_t myRecvOff(const BlockShared* sh) {
  return (sh->dyn.sqeFlags & SQE_RECV_STAGED) ? sh->cs.stagingRecvOff : sh->dyn.recv;
}
// (the offsets the peers posted with their arrival; mine are not posted to myself)
DF_HD const char* sendPtrOf(const BlockShared* sh, int j) { return sh->cs.peerHeap[j] + (j == sh->cs.rank ? mySendOff(sh) : sh->peerSend[j]); }
DF_HD char* recvPtrOf(const BlockShared* sh, int j) { return sh->cs.peerHeap[j] + (j == sh->cs.rank ? myRecvOff(sh) : sh->peerRecv[j]); }

// Schedules in which a user buffer is touched by this rank only use it where it is (no staging copy even when it
// lies outside the symmetric heap): both buffers of the push schedule, the input of a multimem all-gather or
// broadcast, the output of a multimem reduce-scatter.
DF_HD bool rawSend(const CollStatic* c) {
  return c->algo == dfcclAlgoPush || (c->algo == dfcclAlgoNvls && (c->kind == dfcclCollAllGather || c->kind == dfcclCollBroadcast));
}
DF_HD bool rawRecv(const CollStatic* c) { return c->algo == dfcclAlgoPush || (c->algo == dfcclAlgoNvls && c->kind == dfcclCollReduceScatter); }

// Schedules that read or write peers' buffers need the offsets the peers posted.
DF_HD bool needsOffsets(const CollStatic* c) { return c->nranks > 1 && c->algo != dfcclAlgoPush && c->algo != dfcclAlgoNvls; }

// Push schedule: the user's buffers are only touched by this rank, so they are used where they are.
DF_HD const char* pushSendPtr(const BlockShared* sh) {
  return (sh->dyn.sqeFlags & SQE_SEND_STAGED) ? (const char*)(uintptr_t)sh->dyn.send : sh->cs.peerHeap[sh->cs.rank] + sh->dyn.send;
}
DF_HD char* pushRecvPtr(const BlockShared* sh) {
  return (sh->dyn.sqeFlags & SQE_RECV_STAGED) ? (char*)(uintptr_t)sh->dyn.recv : sh->cs.peerHeap[sh->cs.rank] + sh->dyn.recv;
}
// slot that `writer` fills at member `owner` for this epoch's parity
DF_HD char* pushSlot(const BlockShared* sh, int owner, int writer) {
  const CollStatic* c = &sh->cs;
  return c->peerPush[owner] + ((uint64_t)(sh->dyn.epoch & 1u) * c->nranks + writer) * c->pushSlotBytes;
}
// [beg, end) of block b, in the units of the partition
DF_HD void blockRange(const CollStatic* c, int b, uint64_t* beg, uint64_t* end) {
  *beg = umin64(c->total, c->per * (uint64_t)b);
  *end = umin64(c->total, *beg + c->per);
}

// The peers' offsets, one lane of the first warp per peer (the slots hold them until the peers' next arrival).
DF_HD void fetchPeerOffsets(BlockShared* sh, int b) {
  const int n = sh->cs.nranks;
  const FlagSlot* f = sh->cs.myFlags + (uint64_t)b * n;
  for (int j = df_lane(); j < n; j += df_warpsize()) {
    if (j == sh->cs.rank) continue;
    sh->peerSend[j] = offValue(ld_relaxed_sys_u64(&f[j].sendOff));
    sh->peerRecv[j] = offValue(ld_relaxed_sys_u64(&f[j].recvOff));
  }
  df_warp_sync();
}

// What one visit of the data phase moves: the pointer lists, one lane of the first warp per member, and the slice
// [cursor, cursor + slice) of the block's share (slices are multiples of 16 units, so every pointer keeps its 16-byte
// alignment).  A block-wide barrier follows.
DF_HD void buildArgs(BlockShared* sh, int b) {
  const CollStatic* c = &sh->cs;
  DataArgs* a = &sh->args;
  const int n = c->nranks, me = c->rank, lane = df_lane(), ws = df_warpsize();
  const bool push = c->algo == dfcclAlgoPush && n > 1, nvls = c->algo == dfcclAlgoNvls && n > 1;
  if (push && c->kind == dfcclCollAllGather) { if (lane == 0) sh->ctl64 = 0; return; }      // (pushGatherLocal)
  uint64_t beg, end;
  blockRange(c, b, &beg, &end);
  if (c->kind == dfcclCollReduce || (c->kind == dfcclCollAllReduce && n > 1 && !push && c->algo != dfcclAlgoOneShot)) {
    const uint64_t len = end - beg, per = len == c->per ? c->perShard : c->perShardLast;        // my shard of the block's range
    const uint64_t sb = umin64(len, per * (uint64_t)me);
    end = beg + umin64(len, sb + per);
    beg += sb;
  }
  const uint64_t total = end - beg, cur = umin64(sh->dyn.cursor, total);
  uint64_t win = total - cur;
  if (c->sliceUnits && win > c->sliceUnits) win = c->sliceUnits;
  beg += cur;
  const uint64_t in = c->reduces ? beg * (uint64_t)c->esIn : beg, out = c->reduces ? beg * (uint64_t)c->esOut : beg;     // bytes
  const uint64_t piece = c->total * (c->reduces ? (uint64_t)c->esIn : 1);       // bytes of a member's piece of a gathered or scattered array
  int nsrc = 1, ndst = 1, how = c->reduces ? 1 : 0;      // how: 0 copy, 1 reduce, 2 - 4 multimem all-reduce, reduce-scatter, broadcast
  for (int k = lane; k < n; k += ws) {
    int j = me + k;
    if (j >= n) j -= n;
    switch (c->kind) {
      case dfcclCollAllReduce:
        if (push) {                                      // everything is here: my own input plus the slots the peers filled
          a->src[k] = (k == 0 ? pushSendPtr(sh) : (const char*)pushSlot(sh, me, j)) + in;
          if (k == 0) a->dst[0] = pushRecvPtr(sh) + out;
          nsrc = n;
        } else if (nvls) {                               // byte offsets into the arena (symmetric on all members)
          a->src[0] = (const char*)(uintptr_t)(((sh->dyn.sqeFlags & SQE_SEND_STAGED) ? c->nvlsIn : sh->dyn.send) + in);
          a->dst[0] = (char*)(uintptr_t)(((sh->dyn.sqeFlags & SQE_RECV_STAGED) ? c->nvlsOut : sh->dyn.recv) + out);
          how = 2;
        } else if (c->algo == dfcclAlgoOneShot || n == 1) {
          a->src[j] = sendPtrOf(sh, j) + in;
          if (k == 0) a->dst[0] = recvPtrOf(sh, me) + out;
          nsrc = n;
        } else {
          a->src[k] = sendPtrOf(sh, j) + in;
          a->dst[k] = recvPtrOf(sh, j) + out;
          nsrc = ndst = n;
        }
        break;
      case dfcclCollReduce:
        a->src[k] = sendPtrOf(sh, j) + in;
        if (k == 0) a->dst[0] = recvPtrOf(sh, c->root) + out;
        nsrc = n;
        break;
      case dfcclCollReduceScatter:
        if (nvls) {                                      // the switch reduces my block of every member's input (arena); the result stays here
          a->src[0] = (const char*)(uintptr_t)(((sh->dyn.sqeFlags & SQE_SEND_STAGED) ? c->nvlsIn : sh->dyn.send) + (uint64_t)me * piece + in);
          a->dst[0] = pushRecvPtr(sh) + out;
          how = 3;
        } else {
          // my chunk of my own input plus my chunk of every peer's input (push: which they put into their slots here)
          a->src[k] = push ? (k == 0 ? pushSendPtr(sh) + (uint64_t)me * piece : pushSlot(sh, me, j) + (((uint64_t)me * piece) & 15)) + in
                           : sendPtrOf(sh, j) + (uint64_t)me * piece + in;
          if (k == 0) a->dst[0] = (push ? pushRecvPtr(sh) : recvPtrOf(sh, me)) + out;
          nsrc = n;
        }
        break;
      case dfcclCollAllGather:
        if (nvls) {                                      // one multicast store puts my piece into every member's output (arena)
          a->src[0] = pushSendPtr(sh) + in;
          a->dst[0] = (char*)(uintptr_t)(((sh->dyn.sqeFlags & SQE_RECV_STAGED) ? c->nvlsOut : sh->dyn.recv) + (uint64_t)me * piece + out);
          how = 4;
        } else {
          const char* src = sendPtrOf(sh, me) + in;
          const int held = recvPtrOf(sh, me) + (uint64_t)me * piece + in == src ? 1 : 0;        // in place: my own slot already holds it
          if (k == 0) a->src[0] = src;
          if (k >= held) a->dst[k - held] = recvPtrOf(sh, j) + (uint64_t)me * piece + out;
          ndst = n - held;
        }
        break;
      default:                                           // broadcast
        if (nvls) {
          // the root's multicast stores put its buffer into every member's output (arena); the others move nothing and
          // learn from the root's done flag that their output is complete
          a->src[0] = pushSendPtr(sh) + in;
          a->dst[0] = (char*)(uintptr_t)(((sh->dyn.sqeFlags & SQE_RECV_STAGED) ? c->nvlsOut : sh->dyn.recv) + out);
          ndst = me == c->root ? 1 : 0;
          how = 4;
        } else if (k == 0) {
          a->src[0] = sendPtrOf(sh, c->root) + in;
          a->dst[0] = recvPtrOf(sh, me) + out;
          ndst = a->dst[0] == a->src[0] ? 0 : 1;
        }
        break;
    }
  }
  if (lane == 0) {
    a->nsrc = nsrc; a->ndst = ndst; a->n = win; a->scale = c->scale; a->postDiv = c->postDiv;
    sh->ctl64 = cur + win < total ? cur + win : 0;       // the next cursor; 0 = this is the last slice
    sh->ctl1 = how;
    if (c->reduces) sh->stats.bytesReduced += win * c->esIn * nsrc; else sh->stats.bytesCopied += win * ndst;
  }
}

// ---- bounded waits (first warp polls, everybody learns the outcome)
// which: 0 = arrive flags (the pointer lists of the data phase are built while everybody else still waits), 1 = done flags,
// 2 = local trigger word
DF_HD bool boundedWait(BlockShared* sh, RankDev* rd, int b, int which, uint32_t budget) {
  if (df_tid() < df_warpsize()) {
    const int lane = df_lane(), ws = df_warpsize();
    const int n = sh->cs.nranks, me = sh->cs.rank;
    const uint32_t epoch = sh->dyn.epoch;
    // Members on one device post with relaxed stores, and the tags tell whose epoch an offset is; the others' arrival is a
    // release, behind which the offsets are read.
    const bool offsets = which == 0 && needsOffsets(&sh->cs) && sh->cs.oneDevice;
    FlagSlot* mine = sh->cs.myFlags + (uint64_t)b * n;
    uint32_t spins = 0;
    bool ok;
    // At every fourth poll the last lane looks at the ring too, its load on its way with theirs: a wait with a lot of patience ends when
    // there is something else to do, which an entry is not that the block has met and cannot take, and hardly one that a stream has yet to
    // release.  (At every sixteenth where all peers are in the collective already: they are done soon, and another collective's context
    // costs more than that.)  us, all-reduces of bf16 -> fp32 that one stream releases in the same order on all ranks, no look / a look that any
    // entry ends / now: 2 ranks 4 x 1 M 115 / 123 / 114, 4 ranks 141 / 158 / 148, 4 ranks 8 x 500 K 249 / 279 / 264; 2 ranks 8 x 1 M in two orders 283 /
    // 234 / 238 (277 where these entries end no wait, the others then 112, 142, 254).
    const uint32_t often = which == 1 ? 15u : 3u;
    for (;;) {
      bool laneOk = true;
      uint64_t entry = 0, tag = 1;
      if ((spins & often) == often && lane == ws - 1 && !sh->standalone && sh->k.devSq != nullptr && sh->frontier != sh->stuckAt) {
        entry = ld_relaxed_sys_u64(sh->k.devSq[sh->frontier & (sh->k.sqCap - 1)].w);
        tag = sqTag(sh->frontier, sh->k.sqCap);
      }
      if (which == 2) {
        if (lane == 0) laneOk = (int32_t)((uint32_t)ld_relaxed_sys_u64(&sh->k.trigger[sh->loadedColl]) - (uint32_t)sh->dyn.trigger) >= 0;
      } else {
        for (int j = lane; j < n; j += ws) {
          if (j == me) continue;
          if (offsets) {
            uint64_t v, so;
            ld_relaxed_sys_2u64(&mine[j].arrive, &v, &so);
            const uint64_t ro = ld_relaxed_sys_u64(&mine[j].recvOff);
            laneOk = laneOk && v >= epoch && offCurrent(so, epoch) && offCurrent(ro, epoch);
            sh->peerSend[j] = offValue(so); sh->peerRecv[j] = offValue(ro);
          } else {
            laneOk = laneOk && ld_relaxed_sys_u64(which == 0 ? &mine[j].arrive : &mine[j].done) >= epoch;
          }
        }
      }
      bool laneStop = false;
      if ((spins & 255) == 255 && lane == 0) laneStop = abortRequested(&sh->k) || (!sh->standalone && ld_relaxed_sys_u32(&rd->quitting) != 0);      // (the others have left: so does this block)
      if (entry >> 57 == tag && (!((entry >> 48) & SQE_TRIGGERED) || spins + 1 >= pollsBesideTriggers(&sh->k))) laneStop = true;
      ok = df_warp_all(laneOk);
      const bool stop = !df_warp_all(!laneStop);      // uniform: every lane leaves the loop together
      ++spins;
      if (ok || stop || spins >= budget) break;
    }
    // polls are relaxed loads (an acquire at system scope per poll costs a fence each time); the one
    // fence that orders the payload accesses after the flags is paid when the wait succeeds
    if (ok) { if (which == 2) fence_sys(); else fence_members(&sh->cs); }
    df_warp_sync();
    if (ok && which == 0) {
      if (needsOffsets(&sh->cs) && !offsets) fetchPeerOffsets(sh, b);
      buildArgs(sh, b);
    }
    if (lane == 0) { sh->waitOk = ok ? 1 : 0; sh->waitSpins = spins; sh->stats.waitPolls += spins; }
  }
  df_sync();
  return sh->waitOk != 0;
}

// Called by all threads when a wait ran out.  Returns true if the collective must fail now.
DF_HD bool noteStall(BlockShared* sh, RankDev* rd) {
  if (df_tid() == 0) {
    uint64_t now = df_now_ns();
    sh->ctl0 = 0;
    if (sh->standalone ? abortRequested(&sh->k) : (sh->abortSeen != 0)) { sh->dyn.status = ST_ABORTED; sh->ctl0 = 1; }
    else if (sh->dyn.stallSinceNs == 0) { sh->dyn.stallSinceNs = now; sh->dynDirty = 1; }
    else if (sh->k.waitTimeoutNs && now - sh->dyn.stallSinceNs > sh->k.waitTimeoutNs) {
      sh->dyn.status = ST_TIMEOUT; sh->ctl0 = 1; sh->stats.waitTimeouts++;
    }
  }
  df_sync();
  return sh->ctl0 != 0;
}

// `n` bytes by the whole block, four packs of a thread in flight; several of these follow one another without a barrier.
DF_HD void copyOne(const char* src, char* dst, uint64_t n) {
  const int tid = df_tid(), nt = df_nthreads();
  const uint32_t head = (uint32_t)umin64((16u - (uint32_t)((uintptr_t)dst & 15)) & 15u, n);
  const uint32_t shift = (uint32_t)(((uintptr_t)src + head) & 15);
  const uint64_t nPacks = (n - head) / 16;             // (a piece is as long as the limit of the push schedule is set: bytes take 64 bits)
  const char* s = src + head - shift;
#pragma unroll 1
  for (uint64_t p0 = (uint64_t)tid; p0 < nPacks; p0 += 4u * (uint32_t)nt) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint64_t p = p0 + (uint32_t)(u * nt);
      if (p >= nPacks) continue;
      v[u] = ld16(s + p * 16);
      if (shift) v[u] = shiftPack(v[u], ld16(s + p * 16 + 16), shift);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint64_t p = p0 + (uint32_t)(u * nt);
      if (p < nPacks) st16(dst + head + p * 16, v[u]);
    }
  }
  const uint64_t tail0 = head + nPacks * 16;
#pragma unroll 1
  for (uint64_t i = (uint64_t)(nt - 1 - tid); i < head + (n - tail0); i += nt) {
    const uint64_t e = i < head ? i : tail0 + (i - head);
    st_elem((uint8_t*)dst + e, ld_elem((const uint8_t*)src + e));
  }
}

// Push schedule, outgoing half: what the peers need of my input goes into my slot at each of them (block b moves its
// part of the range).  All-reduce: the whole input to everybody.  All-gather: my piece to everybody.
// Reduce-scatter: chunk j of my input to member j.  Ends with a barrier.
DF_HD void pushOut(BlockShared* sh, int b) {
  const CollStatic* c = &sh->cs;
  const int n = c->nranks, me = c->rank;
  uint64_t beg, end;
  blockRange(c, b, &beg, &end);
  const uint64_t unit = c->reduces ? (uint64_t)c->esIn : 1, bytes = (end - beg) * unit;
  beg *= unit;
  if (c->kind == dfcclCollReduceScatter) {
    if (bytes) {
#pragma unroll 1
      for (int k = 1; k < n; ++k) {                // a different chunk for every member: one copy each
        int j = me + k;
        if (j >= n) j -= n;
        // the chunk sits in the slot at the misalignment it has in the input (chunks of odd length start off the
        // 16-byte grid), so that the receiver's sources - its own chunk and the slots - all line up alike
        const uint64_t off = (uint64_t)j * c->total * unit;
        copyOne(pushSendPtr(sh) + off + beg, pushSlot(sh, j, me) + (off & 15) + beg, bytes);
      }
    }
    if (df_tid() == 0) sh->stats.bytesCopied += bytes * (n - 1);
    df_sync();
    return;
  }
  if (df_tid() < df_warpsize()) {
    DataArgs* a = &sh->args;
    for (int k = 1 + df_lane(); k < n; k += df_warpsize()) {
      int j = me + k;
      if (j >= n) j -= n;
      a->dst[k - 1] = pushSlot(sh, j, me) + beg;
    }
    if (df_lane() == 0) {
      a->nsrc = 1; a->ndst = n - 1; a->n = bytes;
      a->src[0] = pushSendPtr(sh) + beg;
      sh->stats.bytesCopied += bytes * (n - 1);
    }
  }
  df_sync();
  if (bytes && n > 1) copy_block(&sh->args);
  df_sync();
}

// Push schedule, all-gather: every member's piece is in its slot here; block b copies its part of each into the
// output (my own piece comes from my input, unless the call is in place).  Pieces are small: no slicing.
DF_HD void pushGatherLocal(BlockShared* sh, int b) {
  const CollStatic* c = &sh->cs;
  const int n = c->nranks, me = c->rank;
  uint64_t beg, end;
  blockRange(c, b, &beg, &end);
  if (beg == end) return;
#pragma unroll 1
  for (int j = 0; j < n; ++j) {
    const char* src = (j == me ? pushSendPtr(sh) : (const char*)pushSlot(sh, me, j)) + beg;
    char* dst = pushRecvPtr(sh) + (uint64_t)j * c->total + beg;
    if (dst == src) continue;                      // in place: my piece already sits where it belongs
    copyOne(src, dst, end - beg);
    if (df_tid() == 0) sh->stats.bytesCopied += end - beg;
  }
}

static DF_HD_NOINLINE bool moveMultimem(const BlockShared* sh) {
  const CollStatic* c = &sh->cs;
  const DataArgs* a = &sh->args;
  const uint64_t in = (uint64_t)(uintptr_t)a->src[0], out = (uint64_t)(uintptr_t)a->dst[0];
  if (sh->ctl1 == 2) return nvlsDispatch(c->inType, c->outType, c->mcHeap, c->nvlsPeers, c->nranks, in, out, a->n, (float)c->scale);
  if (sh->ctl1 == 3) return nvlsDispatchToLocal(c->inType, c->outType, c->mcHeap, c->nvlsPeers, c->nranks, in, a->dst[0], a->n, (float)c->scale);
  nvlsBroadcastBytes(c->mcHeap, c->nvlsPeers, c->nranks, a->src[0], out, a->n);
  return true;
}

// ---- PH_DATA: everybody moves the data of the pointer lists (buildArgs).
// The block's share is moved in slices of `sliceBytes` (0 = all at once): after a slice the cursor is saved and
// the function returns true when more is left, so that the caller can hand the block to another collective and
// come back later - the resumable data phase (reference: slice / offset saved inside one primitive and
// currentStep / gridOffset in the ring loop, src/collectives_ofccl/device/ofccl_prims_simple.h:239-244,326-346,
// ofccl_all_reduce.h:86-93,192-205).  A slice never waits for anybody, so leaving between two slices has no side
// effect beyond the cursor.  `sh->ctl0` tells the caller whether anything else wants the block.
DF_HD bool dataPhase(BlockShared* sh, RankDev* rd, int b) {
  const CollStatic* c = &sh->cs;
  if (c->kind == dfcclCollAllGather && c->algo == dfcclAlgoPush && c->nranks > 1) { pushGatherLocal(sh, b); df_sync(); return false; }
  if (sh->args.n != 0 && sh->args.ndst != 0) {
    const int how = sh->ctl1;
    bool known = true;
    if (how == 1) known = reduce_block(c->inType, c->outType, c->esIn, c->op, &sh->args);
    else if (how == 0) copy_block(&sh->args);
    else known = moveMultimem(sh);
    if (!known && df_tid() == 0) sh->dyn.status = ST_BAD_ARG;
  }
  df_sync();
  const bool more = sh->ctl64 != 0;
  if (more) {
    if (df_tid() == 0) {
      sh->dyn.cursor = sh->ctl64; sh->dynDirty = 1;
      // anything else for this block?  queued collectives, submissions waiting for their stream, or entries of the
      // device ring this block has not consumed yet
      SqSlot next;
      sh->ctl0 = !sh->standalone && (sh->nActive > 1 || sh->nTrig > 0 || sqPeek(&sh->k, sh->frontier, &next)) ? 1 : 0;
    }
    df_sync();
  }
  return more;
}

// ---- staging copies for buffers outside the symmetric heap
// Block b copies exactly the bytes that block b of the peers (or of this rank) touches in
// PH_DATA, because the flags of block b are the only ordering between the two: the same
// partition as dataPhase, element-based for reducing kinds, byte-based for copying kinds.
static DF_HD_NOINLINE void stageCopy(BlockShared* sh, int b, bool in) {
  const CollStatic* c = &sh->cs;
  const uint64_t e = in ? c->esIn : c->esOut;
  const int segs = (in && c->kind == dfcclCollReduceScatter) || (!in && c->kind == dfcclCollAllGather) ? c->nranks : 1;
  const uint64_t segBytes = c->count * e;
  uint64_t beg, end;
  blockRange(c, b, &beg, &end);
  if (c->reduces) { beg *= e; end *= e; }
  for (int s = 0; s < segs; ++s) {
    if (df_tid() == 0) {
      DataArgs* a = &sh->args;
      a->nsrc = 1; a->ndst = 1; a->n = end - beg;
      const uint64_t off = (uint64_t)s * segBytes + beg;
      if (in) { a->src[0] = (const char*)sh->dyn.send + off; a->dst[0] = c->peerHeap[c->rank] + c->stagingSendOff + off; }
      else { a->src[0] = c->peerHeap[c->rank] + c->stagingRecvOff + off; a->dst[0] = (char*)sh->dyn.recv + off; }
      sh->stats.bytesCopied += a->n;
    }
    df_sync();
    if (sh->args.n) copy_multi(&sh->args);
    df_sync();
  }
}

// ---- completion: count blocks; the last one publishes the device flag and the CQE
// `idx`: the place of the host's entry, asked for before the fences so that it is on its way meanwhile.  `early`: a stream may be
// parked on the device flag.
DF_HD void publishCompletion(BlockShared* sh, unsigned long long idx, int coll, uint32_t st, uint32_t epoch, bool early) {
  // The device flag releases a stream of THIS GPU (its wait is a stream memory operation, the consumers are kernels
  // launched behind it): everything the blocks wrote here is ordered before it by a fence of GPU scope, a quarter
  // of the cost of a system-scope one.  (What the blocks wrote into peers' memory was ordered by the fence before
  // their done flags, and this rank's result was complete when every peer's done flag had arrived.)
  if (early) {
    fence_acq_rel_gpu();
    st_relaxed_sys_u64(&sh->k.doneEpoch[coll], ((uint64_t)st << 56) | epoch);
  }
  // the host's entry: a host thread may read the result right after the callback, so the data is ordered system-wide
  fence_acq_rel_sys();
  if (!early) st_relaxed_sys_u64(&sh->k.doneEpoch[coll], ((uint64_t)st << 56) | epoch);
  const uint32_t cap = sh->k.cqCap, gen = (uint32_t)(idx >> log2Of(cap)) + 1u;
  st_relaxed_sys_u64(&sh->k.hostCq[idx & (cap - 1)], cqeEncode(gen, st, (uint32_t)coll));
}

// Thread 0 alone has something to do; no barrier (the next one the block meets is in front of whatever changes the context).
DF_HD void completeColl(BlockShared* sh, RankDev* rd, int b) {
  if (df_tid() != 0) return;
  if (sh->standalone) {                           // stream-ordered kernel: report errors only
    if (sh->dyn.status != ST_OK) sh->k.ctl->pad = sh->dyn.status;
    return;
  }
  const int coll = sh->loadedColl;
  const uint32_t status = sh->dyn.status;
  // the cached copy stays authoritative while the collective is loaded; it reaches global memory when another
  // collective is loaded, when the block parks, or when the next submission of this id is consumed
  sh->stats.collsDone++;
  uint32_t st = status <= ST_BAD_ARG ? status : (uint32_t)ST_TIMEOUT;
  bool last = true;
  if (sh->cs.nBlocks > 1) {                       // one word counts the blocks and carries their verdicts
    fence_acq_rel_gpu();
    const uint32_t mine = doneWord(st), all = atomic_add_u32(&sh->k.doneCount[coll], mine) + mine;
    last = (all & 0xffu) == (uint32_t)sh->cs.nBlocks;
    st = doneVerdict(all);
  }
  if (last) {
    const unsigned long long idx = atomic_add_u64((unsigned long long*)&rd->devCqTail, 1ull);
    if (sh->cs.nBlocks > 1) atomic_exch_u32(&sh->k.doneCount[coll], 0u);
    publishCompletion(sh, idx, coll, st, sh->dyn.epoch, (sh->dyn.sqeFlags & SQE_TRIGGERED) != 0);
  }
  trace(sh, rd, b, TR_DONE, coll);
}

// The first phase from `phase` on that has something to do for the loaded submission (a phase change costs two
// block-wide barriers, a small collective would otherwise spend more time changing phases than moving data).
// (Comparisons in the order of the phases: a jump table is a load from constant memory that a block meets cold.)
DF_HD int nextPhase(const BlockShared* sh, int phase) {
  const CollStatic* c = &sh->cs;
  const int n = c->nranks, me = c->rank;
  if (phase <= PH_COPY_IN && (sh->dyn.sqeFlags & SQE_SEND_STAGED) && !rawSend(c) && !(c->kind == dfcclCollBroadcast && me != c->root)) return PH_COPY_IN;
  if (phase <= PH_WAIT_ARRIVE && n > 1) return phase < PH_POST_ARRIVE ? PH_POST_ARRIVE : phase;
  if (phase <= PH_DATA) return PH_DATA;
  if (phase <= PH_WAIT_DONE && n > 1 && c->algo != dfcclAlgoPush) return phase;
  if (phase <= PH_COPY_OUT && (sh->dyn.sqeFlags & SQE_RECV_STAGED) && !rawRecv(c) && !(c->kind == dfcclCollReduce && me != c->root)) return PH_COPY_OUT;
  return PH_COMPLETE;
}

// A wait of the loaded collective with its adaptive budget.  The budget is what the scheduler grants or, if larger and nothing else
// is queued or may be released, the patience this submission has earned: after a wait succeeded within s polls the next waits of the same
// submission may spend factor x s polls (capped), because a collective whose peers are demonstrably in it is worth
// staying with (reference: RECV_SUCCESS_FACTOR, src/collectives_ofccl/device/ofccl_prims_simple.h:79-88,143-151).  Beside others the
// oldest of the queue has NUM_TRY_TASKQ_HEAD times the budget if a stream released it.
DF_HD bool patientWait(BlockShared* sh, RankDev* rd, int b, int which, uint32_t budget) {
  uint32_t eff = budget;
  if (sh->standalone || (sh->nActive <= 1 && sh->nTrig == 0)) {
    if (sh->dyn.patience > eff) eff = sh->dyn.patience;
  } else if (sh->nActive > 1 && (sh->dyn.sqeFlags & SQE_TRIGGERED) && sh->active[0] == sh->loadedColl) eff = budget * sh->k.headTries;
  const bool ok = boundedWait(sh, rd, b, which, eff);
  if (ok && df_tid() == 0) {
    sh->dyn.stallSinceNs = 0;
    if (!sh->standalone && sh->k.recvSuccessFactor) {
      uint64_t p = (uint64_t)sh->waitSpins * sh->k.recvSuccessFactor;
      const uint64_t cap = (uint64_t)sh->k.spinBudget * 64u;
      if (p > cap) p = cap;
      if (p > sh->dyn.patience) { sh->dyn.patience = (uint32_t)p; sh->dynDirty = 1; }
    }
  }
  return ok;
}

// Run the loaded-or-to-be-loaded collective until it completes, a wait runs out (RC_STALLED) or its data phase
// reaches a slice boundary while other work is queued (RC_YIELD).
// `budget` is the number of polls one wait may spend.
// `*moved` is set when at least one phase (or slice) was left behind during this visit.
// The phase lives in a register of every thread: a visit reads it when it begins, and thread 0 writes it back when it ends
// (every way out has met a barrier since the read), so that a change of phase costs no barrier of its own.
// What bounds a small collective here is instructions, barriers and round trips to L2 one behind the other, in one block.  Hence
// the phase in a register, the rank's constants in shared memory, the partition worked out at registration, the pointer lists built
// by one lane per member in front of the barrier that ends the wait, small bodies (datapath.h), one atomic for the blocks' count and
// verdicts, comparisons instead of jump tables, and no fence that nobody waits for.  Among four ranks of a device, submitted and
// awaited on the host, before / with all of these and calls that do not go through ctypes, us: 509 bf16 33.9 / 19.8, 25 MiB
// bf16 -> fp32 97.9 / 81.2, a ragged reduce-scatter and all-gather 90.7 / 66.5, 24 mixed collectives in four orders 295 / 211; since, with
// other bodies of the sums (datapath.h) and shorter waits (daemon_impl.h), 76.2, 54.3 and 147.
DF_HD int runColl(BlockShared* sh, RankDev* rd, int b, int coll, uint32_t budget, bool* moved) {
  if (!sh->standalone) loadColl(sh, rd, b, coll);
  const CollStatic* c = &sh->cs;
  const int rb = sh->standalone ? b : relBlock((int)sh->k.nBlocks, c, b);      // my index among this collective's blocks
  const int n = c->nranks, me = c->rank;
  const int tid = df_tid();
  const bool warp0 = tid < df_warpsize();
  int phase = sh->dyn.phase;
  const int entryPhase = phase;
  bool listed = false;                                       // the pointer lists are up to date
  bool fetch = phase == PH_DATA && needsOffsets(c);          // resumed between two slices: another collective's offsets may stand here
  int rc = -1;
  // each phase that is due leads to a later one, or (a slice of the data) stays
  do {
    if (phase == PH_TRIGGER) {
      // (the daemon releases stream-ordered submissions from its trigger list and enters at PH_COPY_IN; this
      // phase serves entries that were parked here by an earlier instance)
      if ((sh->dyn.sqeFlags & SQE_TRIGGERED) && !boundedWait(sh, rd, rb, 2, sh->standalone ? budget : 1u)) {
        if (!noteStall(sh, rd)) { rc = RC_STALLED; break; }
        phase = PH_COMPLETE;
      } else {
        if (tid == 0) { sh->dyn.stallSinceNs = 0; trace(sh, rd, b, TR_START, coll); }
        phase = nextPhase(sh, PH_COPY_IN);
      }
    }
    if (phase == PH_COPY_IN) {
      if ((sh->dyn.sqeFlags & SQE_SEND_STAGED) && !rawSend(c) && !(c->kind == dfcclCollBroadcast && me != c->root)) stageCopy(sh, rb, true);
      phase = nextPhase(sh, PH_POST_ARRIVE);
    }
    if (phase == PH_POST_ARRIVE) {
      const bool pushed = c->algo == dfcclAlgoPush && n > 1;
      if (pushed) pushOut(sh, rb);                           // the payload travels ahead of the arrival flag: stores, a fence, the flag
      if (warp0) {
        if (pushed || (sh->dyn.sqeFlags & SQE_SEND_STAGED)) fence_members(c);        // what the block has stored, a barrier ago
        const uint32_t epoch = sh->dyn.epoch;
        const uint64_t so = offTagged(mySendOff(sh), epoch), ro = offTagged(myRecvOff(sh), epoch);
        for (int j = tid; j < n; j += df_warpsize()) {
          if (j == me) continue;
          FlagSlot* s = c->peerFlags[j] + (uint64_t)rb * n + me;
          if (!pushed) { st_relaxed_sys_u64(&s->sendOff, so); st_relaxed_sys_u64(&s->recvOff, ro); }        // (not used by the push schedule)
          if (c->oneDevice || pushed) st_relaxed_sys_u64(&s->arrive, epoch); else st_release_sys_u64(&s->arrive, epoch);
        }
      }
      phase = PH_WAIT_ARRIVE;                                // the warp that posted is the one that polls
    }
    if (phase == PH_WAIT_ARRIVE) {
      if (n > 1 && !patientWait(sh, rd, rb, 0, budget)) {
        if (!noteStall(sh, rd)) {
          if (tid == 0) trace(sh, rd, b, TR_STALL, coll);
          rc = RC_STALLED;
          break;
        }
        phase = PH_COMPLETE;
      } else {
        listed = n > 1;
        if (tid == 0) trace(sh, rd, b, TR_ARRIVED, coll);
        phase = PH_DATA;
      }
    }
    if (phase == PH_DATA) {
      if (phase != entryPhase) *moved = true;
      if (!listed) {
        if (warp0 && fetch) fetchPeerOffsets(sh, rb);
        fetch = false;
        if (warp0) buildArgs(sh, rb);
        df_sync();
      }
      listed = false;
      if (tid == 0) trace(sh, rd, b, TR_DATA_BEGIN, coll);
      const bool more = dataPhase(sh, rd, rb);               // ends with a barrier
      if (tid == 0) trace(sh, rd, b, TR_DATA_END, coll);
      if (more) {                                            // the cursor is saved; the phase stays PH_DATA
        *moved = true;
        if (sh->ctl0) {
          if (tid == 0) { sh->stats.yields++; trace(sh, rd, b, TR_YIELD, coll); }
          rc = RC_YIELD;
        }
        continue;
      }
      // (push schedule: no done handshake - nobody reads my buffers and my slots are not reused before the
      // peers' next-but-one call)
      phase = nextPhase(sh, PH_POST_DONE);
    }
    if (phase == PH_POST_DONE) {
      if (n > 1 && warp0) {
        // all payload stores of this block were issued before the barrier at the end of the data phase; a fence of
        // the lanes that post makes them visible to the members before any done flag is
        fence_members(c);
        const uint64_t epoch = sh->dyn.epoch;
        for (int j = tid; j < n; j += df_warpsize())
          if (j != me) st_relaxed_sys_u64(&(c->peerFlags[j] + (uint64_t)rb * n + me)->done, epoch);
      }
      phase = PH_WAIT_DONE;
    }
    if (phase == PH_WAIT_DONE) {
      if (n > 1 && !patientWait(sh, rd, rb, 1, budget)) {
        if (!noteStall(sh, rd)) {
          if (tid == 0) trace(sh, rd, b, TR_STALL, coll);
          rc = RC_STALLED;
          break;
        }
        phase = PH_COMPLETE;
      } else {
        if (tid == 0) trace(sh, rd, b, TR_PEERS_DONE, coll);
        phase = nextPhase(sh, PH_COPY_OUT);
      }
    }
    if (phase == PH_COPY_OUT) {
      if ((sh->dyn.sqeFlags & SQE_RECV_STAGED) && !rawRecv(c) && !(c->kind == dfcclCollReduce && me != c->root)) stageCopy(sh, rb, false);
      phase = PH_COMPLETE;
    }
    completeColl(sh, rd, b);
    rc = RC_DONE;
  } while (rc < 0);
  if (phase != entryPhase) *moved = true;
  if (tid == 0) { sh->dyn.phase = phase; sh->dynDirty = 1; }
  return rc;
}

}  // namespace dfccl
