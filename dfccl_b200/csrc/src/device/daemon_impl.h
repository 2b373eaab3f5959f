// Per-block scheduler of the persistent daemon.
//
// Every block of a rank runs daemonBlockMain independently; nothing in here makes
// one block of a GPU wait for another block of the same GPU.  Each block
//   1. finds new submissions in the device-resident ring (one warp per rank copies
//      them there from the host's ring: no other warp reads host memory),
//   2. consumes every entry of that ring in order (its own frontier), and
//      appends the collectives it takes part in (relative block index < nBlocks of the
//      collective) to its task queue,
//   3. walks the task queue: runs each collective until it finishes or a bounded
//      wait gives up, in which case the collective stays queued and the next one
//      is loaded - the preemption that makes any per-rank issue order deadlock-free,
//   4. leaves voluntarily when it has been idle (or only stalled) for long enough,
//      parking its frontier and task queue in global memory for the next launch.
// Same responsibilities as the reference's daemonKernel loop
// (src/collectives_ofccl/device/enqueue_ofccl_dev.cu:1026-1483: sqRead :85-173,
// checkSQ7TidyTaskQ :491-627, traverseTaskQ :922-1023, voluntary quit :1107-1117,
// state save :1374-1480), with a device-resident queue mirror, a trigger list for
// submissions that wait for their stream (polled without loading any context),
// time-based instead of count-based quit thresholds and a two-integer cursor per
// parked collective.
#pragma once
#include "engine.h"

namespace dfccl {

// The service warp of a rank's first block: copies new entries of the pinned ring into the device ring, up to eight at a
// time (one lane per word), until the block leaves.  Runs beside the block's scheduler and data phases, so that the other
// blocks of the rank find their work whatever this one is doing.
DF_HD void serviceMain(BlockShared* sh, RankDev* rd) {
#if DF_DEVICE_CODE
  const int lane = df_lane();
  uint64_t head = rd->svcHead;
  const uint32_t cap = rd->sqCap;
  for (;;) {
    const uint64_t index = head + (lane >> 2);
    const uint64_t at = (index & (cap - 1)) * 4 + (lane & 3);
    const uint64_t w = ld_relaxed_sys_u64((const volatile uint64_t*)rd->hostSq + at);
    const uint32_t bad = ~__ballot_sync(0xffffffffu, (w >> 57) == sqTag(index, cap));
    const int whole = (bad ? __ffs(bad) - 1 : 32) >> 2;          // entries from `head` on of which every word is there
    if (whole == 0) {
      if (__any_sync(0xffffffffu, sh->svcStop != 0)) break;        // one decision for the warp: the lanes meet in the vote above
      continue;
    }
    // What the host wrote before it published these entries (payloads in memory it writes itself) comes before whatever a
    // block does because of them: the host's release store, this fence, and the block's own fence of GPU scope make the
    // chain.  (One microsecond: 1 KB among four ranks 33.0 us without it, 34.2 with; with acquiring polls and releasing stores
    // instead the same.)
    fence_acq_rel_sys();
    if (lane < 4 * whole) st_relaxed_sys_u64((volatile uint64_t*)rd->devSq + at, w);
    head += whole;
  }
  if (lane == 0) rd->svcHead = head;
#endif
}

// Consume new entries of the device ring.  Thread 0 only.  Returns the number consumed.
// A submission that waits for its stream goes to the trigger list, everything else to the task queue.
// `slot` and `next`: the first two entries, looked at together (a lone entry then costs no second round trip).
DF_HD int consumeSubmissions(BlockShared* sh, RankDev* rd, int b, SqSlot slot, SqSlot next, bool haveNext) {
  int got = 0;
  for (bool have = true; have; slot = next, have = haveNext, haveNext = have && sqPeek(&sh->k, sh->frontier + 1, &next)) {
    const Sqe q = sqDecode(slot);
    if (q.flags & SQE_QUIT) { sh->quit = 2; break; }       // the frontier stays on the quit entry
    const int coll = q.collId;
    bool mine = false;
    if (coll >= 0 && (uint32_t)coll < sh->k.maxColls) {
      const uint32_t m = sh->meta[coll];
      int r = b - (int)((m >> 8) & 0xffu);
      if (r < 0) r += (int)sh->k.nBlocks;
      mine = (m & DF_META_VALID) && r < (int)(m & 0xffu);
    }
    if (mine) {
      // A stream-ordered caller may publish the next submission of a collective while this block
      // still runs the previous one.  The entry is never dropped: consumption stops here and
      // resumes once the running submission has completed.
      const bool full = (q.flags & SQE_TRIGGERED) ? sh->nTrig >= DF_MAX_ACTIVE : sh->nActive >= DF_MAX_ACTIVE;   // (cannot happen: one outstanding submission per id)
      if (full || (sh->busy[coll >> 5] & (1u << (coll & 31)))) { sh->stuckAt = sh->frontier; break; }
    }
    ++sh->frontier;
    ++got;
    sh->stats.sqesSeen++;
    if (!mine) continue;
    sh->busy[coll >> 5] |= 1u << (coll & 31);
    CollDyn d;
    d.send = q.send; d.recv = q.recv; d.trigger = q.trigger; d.cursor = 0;
    d.epoch = q.epoch; d.sqeFlags = q.flags; d.status = ST_OK; d.stallSinceNs = 0; d.patience = 0; d.pad = 0;
    d.phase = (q.flags & SQE_TRIGGERED) ? PH_TRIGGER : PH_COPY_IN;          // runColl skips ahead to the first phase that has work
    if (sh->loadedColl == coll && !(q.flags & (SQE_TRIGGERED | SQE_NEW_STATIC))) { sh->dyn = d; sh->dynDirty = 1; }   // its context is still here
    else {
      if (sh->loadedColl == coll) { sh->loadedColl = -1; sh->dynDirty = 0; }                          // re-armed in global memory: drop the cached copy
      sh->k.dyn[(uint64_t)b * sh->k.maxColls + coll] = d;
    }
    trace(sh, rd, b, TR_SQE, coll);
    if (q.flags & SQE_TRIGGERED) {
      sh->trigColl[sh->nTrig] = (uint16_t)coll; sh->trigVal[sh->nTrig] = q.trigger; ++sh->nTrig;
    } else {
      sh->actWait[sh->nActive] = 0;
      sh->active[sh->nActive++] = (uint16_t)coll;
      trace(sh, rd, b, TR_START, coll);
    }
  }
  if (got) fence_acq_rel_gpu();                            // the entries, before anything that is read because of them
  return got;
}

// How far this block has come, for the host's flow control (it reads this when its ring looks full).  A store across PCIe that
// the next fence of system scope would wait for, so it goes out when the block has nothing to do, or a quarter of the ring behind.
DF_HD void reportFrontier(BlockShared* sh, int b, bool idle) {
  if (sh->frontier == sh->frontierSeen || !(idle || sh->frontier - sh->frontierSeen >= sh->k.sqCap / 4)) return;
  st_relaxed_sys_u64(&sh->k.hostFrontier[b], sh->frontier);
  sh->frontierSeen = sh->frontier;
}

// Look at the trigger words of every submission that waits for its stream: one thread per entry, no context is
// loaded.  Released ones join the task queue in list order.  Everybody calls it; returns the number released.
DF_HD uint32_t pollTriggers(BlockShared* sh, RankDev* rd, int b) {
  const int tid = df_tid(), nt = df_nthreads();
  const uint32_t nTrig = sh->nTrig;
  if (tid == 0) sh->trigFired = 0;
  df_sync();
  for (uint32_t i = tid; i < nTrig; i += nt) {
    const uint32_t have = (uint32_t)ld_relaxed_sys_u64(&sh->k.trigger[sh->trigColl[i]]);
    if ((int32_t)(have - sh->trigVal[i]) >= 0) { sh->trigColl[i] |= 0x8000u; atomic_add_u32(&sh->trigFired, 1u); }
  }
  df_sync();
  const uint32_t fired = sh->trigFired;
  if (fired && tid == 0) {
    fence_sys();                     // what the stream's producers wrote, before anything this block does with it
    uint32_t w = 0;
    for (uint32_t i = 0; i < nTrig; ++i) {
      const uint16_t e = sh->trigColl[i];
      if (e & 0x8000u) {
        const int coll = e & 0x7fff;
        sh->k.dyn[(uint64_t)b * sh->k.maxColls + coll].phase = PH_COPY_IN;
        if (sh->nActive < DF_MAX_ACTIVE) { sh->actWait[sh->nActive] = 0; sh->active[sh->nActive++] = (uint16_t)coll; }
        trace(sh, rd, b, TR_START, coll);
      } else { sh->trigColl[w] = e; sh->trigVal[w] = sh->trigVal[i]; ++w; }
    }
    sh->nTrig = w;
  }
  if (fired) df_sync();
  return fired;
}

// Readiness scan: one thread per parked entry of the task queue reads that collective's flag words of this block
// (n loads of local memory) and marks the entry for a visit when every peer has posted the epoch the entry waits
// for.  No context is loaded and nobody spins: a queue of stalled collectives costs one scan per pass instead of a
// context switch and a polling budget each.  Everybody calls it; returns the number of entries that became ready.
DF_HD uint32_t scanParked(BlockShared* sh, RankDev* rd, int b) {
  const int tid = df_tid(), nt = df_nthreads();
  const uint32_t nAct = sh->nActive;                       // (nReady: cleared at the end of the last pass)
  for (uint32_t i = tid; i < nAct; i += nt) {
    const uint32_t w = sh->actWait[i];
    if (w == 0) continue;
    const int coll = sh->active[i];
    if (coll == 0xffff) continue;
    const CollStatic* c = &sh->k.colls[coll];
    const int n = c->nranks, me = c->rank;
    const FlagSlot* f = c->myFlags + (uint64_t)relBlock((int)sh->k.nBlocks, c, b) * n;
    // (the collective whose context is loaded may have been submitted again since that was last saved)
    const uint64_t epoch = sh->loadedColl == coll ? sh->dyn.epoch : sh->k.dyn[(uint64_t)b * sh->k.maxColls + coll].epoch;
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      if (j == me) continue;
      ok = ok && ld_relaxed_sys_u64(w == 1 ? &f[j].arrive : &f[j].done) >= epoch;
    }
    if (ok) { sh->actWait[i] = 0; atomic_add_u32(&sh->nReady, 1u); }
  }
  df_sync();
  return sh->nReady;
}

DF_HD void blockRestore(BlockShared* sh, RankDev* rd, int b) {
  const int tid = df_tid(), nt = df_nthreads();
  BlockSaved* sv = &rd->saved[b];
  if (tid == 0) {
    sh->k = *rd;
    sh->nParked = 0; sh->nReady = 0; sh->frontierSeen = sv->frontier; sh->stuckAt = ~0ull;
    sh->loadedColl = -1; sh->standalone = 0; sh->dynDirty = 0; sh->quit = 0; sh->abortSeen = 0; sh->ctl1Full = 0;
    sh->frontier = sv->frontier; sh->nActive = sv->nActive; sh->nTrig = sv->nTrig;
    DevStats z = {};
    sh->stats = z;
    sv->exited = 0;
  }
  for (uint32_t i = tid; i < rd->maxColls; i += nt) sh->meta[i] = rd->meta[i];
  for (uint32_t i = tid; i < DF_MAX_COLLS / 32; i += nt) sh->busy[i] = 0;
  df_sync();
  for (uint32_t i = tid; i < sh->nActive; i += nt) { sh->active[i] = sv->active[i]; sh->actWait[i] = 0; }    // everything gets a visit first
  for (uint32_t i = tid; i < sh->nTrig; i += nt) { sh->trigColl[i] = sv->trigColl[i]; sh->trigVal[i] = sv->trigVal[i]; }
  df_sync();
  if (tid == 0) {                                        // what is queued is being worked on
    for (uint32_t i = 0; i < sh->nActive; ++i) if (sh->active[i] != 0xffff) sh->busy[sh->active[i] >> 5] |= 1u << (sh->active[i] & 31);
    for (uint32_t i = 0; i < sh->nTrig; ++i) sh->busy[sh->trigColl[i] >> 5] |= 1u << (sh->trigColl[i] & 31);
  }
  df_sync();
}

DF_HD void blockPark(BlockShared* sh, RankDev* rd, int b) {
  const int tid = df_tid(), nt = df_nthreads();
  if (b == 0 && rd->hostSq) {                              // what the service warp copied is in the ring, its position saved
    if (tid == 0) sh->svcStop = 1;
    df_sync_service();
  }
  saveLoaded(sh, rd, b);
  BlockSaved* sv = &rd->saved[b];
  for (uint32_t i = tid; i < sh->nActive; i += nt) sv->active[i] = sh->active[i];
  for (uint32_t i = tid; i < sh->nTrig; i += nt) { sv->trigColl[i] = sh->trigColl[i]; sv->trigVal[i] = sh->trigVal[i]; }
  df_sync();
  if (tid == 0) {
    reportFrontier(sh, b, true);
    sv->frontier = sh->frontier; sv->nActive = sh->nActive; sv->nTrig = sh->nTrig;
    // fold this launch's counters into the totals the host reads
    DevStats* g = &rd->stats[b];
    g->ctxSwitches += sh->stats.ctxSwitches; g->ctxSaves += sh->stats.ctxSaves; g->ctxLoads += sh->stats.ctxLoads;
    g->waitPolls += sh->stats.waitPolls; g->waitTimeouts += sh->stats.waitTimeouts;
    g->bytesReduced += sh->stats.bytesReduced; g->bytesCopied += sh->stats.bytesCopied;
    g->totalSwitchNs += sh->stats.totalSwitchNs; g->sqesSeen += sh->stats.sqesSeen; g->collsDone += sh->stats.collsDone;
    g->visits += sh->stats.visits; g->yields += sh->stats.yields; g->passes += sh->stats.passes;
    g->nsTriggers += sh->stats.nsTriggers; g->nsWalk += sh->stats.nsWalk; g->nsQueues += sh->stats.nsQueues;
    if (sh->stats.maxSwitchNs > g->maxSwitchNs) g->maxSwitchNs = sh->stats.maxSwitchNs;
    trace(sh, rd, b, TR_QUIT, (int)sh->quit);
    fence_sys();
    sv->exited = 1;
    uint32_t prev = atomic_add_u32(&rd->exitedBlocks, 1u);
    if (prev + 1 == rd->nBlocks) {                     // last block of this rank out: tell the host
      atomic_exch_u32(&rd->exitedBlocks, 0u);
      st_release_sys_u32(&rd->quitting, 0u);
      if (sh->quit == 2) ctl_store(&rd->ctl->finalQuit, 1);
      if (sh->quit == 1) rd->ctl->voluntaryQuits = rd->ctl->voluntaryQuits + 1;
      fence_sys();
      st_release_sys_u32(&rd->ctl->alive, 0u);
    }
  }
}

DF_HD void daemonBlockMain(RankDev* rd, int b, BlockShared* sh) {
  const int tid = df_tid();
  if (df_is_service()) {
    if (b == 0 && rd->hostSq) { df_sync_service(); serviceMain(sh, rd); df_sync_service(); }
    return;
  }
  if (b == 0 && rd->hostSq) {
    if (tid == 0) sh->svcStop = 0;
    df_sync_service();
  }
  blockRestore(sh, rd, b);
  if (tid == 0) trace(sh, rd, b, TR_LAUNCH, 0);
  uint64_t lastUseful = df_now_ns();     // only thread 0's copies of these are ever consulted
  const uint64_t bornNs = lastUseful;
  uint64_t lastSlowCheck = 0, lastFullPass = 0;
  uint32_t winding = 0;
  uint32_t idleBackoff = 32;
  uint64_t tPass = lastUseful;           // when this pass began

  for (;;) {
    // ---- 0. submissions waiting for their stream (every value steering control flow here is block-uniform)
    bool progressed = false;
    if (sh->nTrig) {
      if (pollTriggers(sh, rd, b)) progressed = true;
      if (tid == 0) { const uint64_t t = df_now_ns(); sh->stats.nsTriggers += t - tPass; tPass = t; }
    }
    // ---- 1. task queue traversal: parked entries are skipped unless the scan found their flags ready; now and then
    // every entry is visited all the same, so that a wait that will never succeed reaches its time limit
    const uint32_t nAct = sh->nActive;
    if (nAct) {
      const bool lone = nAct == 1;
      if (!lone && sh->nParked && scanParked(sh, rd, b)) progressed = true;
      const bool fullPass = sh->ctl1Full != 0;
      for (uint32_t i = 0; i < nAct; ++i) {
        const int coll = sh->active[i];
        if (coll == 0xffff) continue;
        if (sh->actWait[i] && !fullPass && !lone) continue;
        // With nothing else queued there is nothing to switch to: the block stays with the collective, whose wait ends when something else is
        // submitted (boundedWait), or after a while beside submissions that a stream may release.
        // With other collectives queued a wait looks twice: the scan looks at the flags of all that are parked at once, and a block that
        // goes on posts the arrivals its peers wait for.  us, 24 mixed collectives of 1 K to 1 M values in four orders / 16 up to 256 K in
        // two / 30 up to 64 K in four: 211 / 94 / 115 where the oldest had twenty polls, the others four, and a submission did not end a
        // wait (of up to 110 us, alone); 147 / 90 / 100 now, with four polls 159 / 78 / 104 against 147 / 73 / 102, eight 172 / 83 / 105.
        // What streams release comes in program order as a rule, the same on all ranks: there the oldest has its tries (2 ranks, 4 x 1 M bf16 ->
        // fp32 by one stream 117.6 -> 114.5, published ahead 126 -> 121; more polls, the same).
        const uint32_t crowd = (sh->k.spinBudget + 15u) / 16u;
        const uint32_t budget = !lone ? crowd : sh->nTrig ? pollsBesideTriggers(&sh->k) : sh->k.spinBudget * sh->k.headTries;
        bool moved = false;
        int rc = runColl(sh, rd, b, coll, budget, &moved);
        if (rc == RC_DONE || rc == RC_YIELD || moved) progressed = true;
        if (tid == 0) {
          sh->stats.visits++;
          if (rc == RC_DONE) { sh->active[i] = 0xffff; sh->busy[coll >> 5] &= ~(1u << (coll & 31)); }
          sh->actWait[i] = rc == RC_STALLED ? (sh->dyn.phase == PH_WAIT_ARRIVE ? 1 : sh->dyn.phase == PH_WAIT_DONE ? 2 : 0) : 0;
        }
        // a collective released by its stream should not wait for a walk over a long queue
        if (sh->nTrig && i + 1 < nAct && pollTriggers(sh, rd, b)) progressed = true;
      }
    }
    df_sync();
    // ---- 2. compaction, new submissions, idle decision: thread 0 decides, everybody obeys
    if (tid == 0) {
      sh->stats.passes++;
      // the words of global memory this section looks at: on their way together
      const uint32_t left = ld_relaxed_sys_u32(&rd->quitting);
      SqSlot slot, next;
      bool haveNext = sqPeek(&sh->k, sh->frontier + 1, &next), have = sqPeek(&sh->k, sh->frontier, &slot);
      // with nothing else to do a look at the ring costs a round trip to L2, a pass several
      if (!progressed && sh->nActive == 0 && sh->nTrig == 0)
        for (int i = 0; i < 8 && !have; ++i) have = sqPeek(&sh->k, sh->frontier, &slot);
      uint32_t w = 0, parked = 0;
      for (uint32_t i = 0; i < sh->nActive; ++i) if (sh->active[i] != 0xffff) { sh->active[w] = sh->active[i]; sh->actWait[w] = sh->actWait[i]; parked += sh->actWait[i] != 0; ++w; }
      sh->nActive = w; sh->nParked = parked; sh->nReady = 0;
      const uint64_t now = df_now_ns();
      sh->ctl1Full = 0;
      if (now - lastFullPass > 2000000) { sh->ctl1Full = 1; lastFullPass = now; }     // every 2 ms: visit parked entries too
      sh->stats.nsWalk += now - tPass;
      // The abort request is sampled every 20 us.
      const bool slow = now - lastSlowCheck > 20000;
      if (slow) {
        sh->abortSeen = abortRequested(&sh->k) ? 1u : 0u;
        lastSlowCheck = now;
      }
      // once one block of this rank has left voluntarily the others take no new work and follow as
      // soon as they cannot progress: a collective needs all its blocks, so the relaunch comes sooner
      winding = left;
      if (have && winding) sh->stuckAt = sh->frontier;
      else if (have && consumeSubmissions(sh, rd, b, slot, next, haveNext) > 0) progressed = true;
      reportFrontier(sh, b, !progressed);
      if (sh->abortSeen) sh->quit = 3;
      else if (sh->k.maxLifetimeNs && now - bornNs > sh->k.maxLifetimeNs && !sh->quit) {
        // safety net: no instance of the daemon outlives this, whatever its state; the host relaunches it
        sh->quit = 1;
        st_release_sys_u32(&rd->quitting, 1u);
      }
      else if (progressed) lastUseful = now;
      // only waiting for streams to release submissions: the host relaunches the daemon when a trigger fires, so by
      // default it leaves as quickly as when idle; a caller whose releases come in quick succession (the buckets
      // of a captured backward pass) can ask it to stay for longer and save the relaunches
      else if (!sh->quit && (winding || now - lastUseful > (sh->nActive ? sh->k.stallQuitNs : sh->nTrig ? sh->k.trigQuitNs : sh->k.idleQuitNs))) {
        // a stream parked on one of this context's completion words must not depend on a host thread's
        // relaunch: while the host holds the instance it only leaves by age (or with the others)
        if (!winding && ctl_load(&sh->k.ctl->hold)) lastUseful = now;
        else {
          sh->quit = 1;
          st_release_sys_u32(&rd->quitting, 1u);
        }
      }
      sh->ctl0 = progressed ? 1 : 0;
      tPass = progressed ? now : df_now_ns();              // (with work at hand the section is short, and the clock a slow read)
      sh->stats.nsQueues += tPass - now;
    }
    df_sync();
    if (sh->quit) break;
    if (sh->ctl0) idleBackoff = 32;
    else if (sh->nActive == 0 && sh->nTrig == 0) {            // nothing to do: poll gently
      df_backoff(idleBackoff);
      if (idleBackoff < 128) idleBackoff *= 2;             // (what it waits for longer, a new submission is seen later)
    }
  }
  blockPark(sh, rd, b);
}

// Stream-ordered execution of ONE collective by a plain (non-persistent) kernel: the
// same phases, but a wait that runs out is simply retried until the time limit.
DF_HD void standaloneBlockMain(RankDev* rd, int b, BlockShared* sh, const CollStatic* cs, uint64_t send, uint64_t recv,
                               uint32_t epoch, uint32_t sqeFlags) {
  if (df_is_service()) return;
  const int tid = df_tid(), nt = df_nthreads();
  {
    const uint4* s = (const uint4*)cs;
    uint4* d = (uint4*)&sh->cs;
    for (int i = tid; i < (int)(sizeof(CollStatic) / 16); i += nt) d[i] = s[i];
  }
  if (tid == 0) {
    sh->k = *rd;
    sh->loadedColl = 0; sh->standalone = 1; sh->dynDirty = 0; sh->quit = 0; sh->abortSeen = 0;
    DevStats z = {};
    sh->stats = z;
    CollDyn d = {};
    // epoch 0 = take it from the device: one more than the collectives this communicator has finished
    d.send = send; d.recv = recv; d.epoch = epoch ? epoch : rd->saEpoch + 1u; d.phase = PH_COPY_IN; d.sqeFlags = sqeFlags; d.status = ST_OK;
    sh->dyn = d;
  }
  df_sync();
  for (;;) {
    bool moved = false;
    if (runColl(sh, rd, b, 0, 4096u, &moved) == RC_DONE) break;
    df_sync();                            // the phase it left is read again
  }
  if (epoch == 0) {                       // the last block out publishes the new count (every block has read the old one by now)
    df_sync();
    if (tid == 0) {
      const uint32_t mine = sh->dyn.epoch;
      if (atomic_add_u32(&rd->exitedBlocks, 1u) + 1u == (uint32_t)sh->cs.nBlocks) {
        atomic_exch_u32(&rd->exitedBlocks, 0u);
        rd->saEpoch = mine;
        fence_sys();
      }
    }
  }
}

}  // namespace dfccl
