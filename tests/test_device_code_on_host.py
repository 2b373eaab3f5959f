"""Parts of the device code compiled for the host by themselves, where the sizes or states they are about cannot be reached through
a communicator on this machine."""
import subprocess

import pytest

from dfccl_b200 import _build


def run_on_host(tmp_path, body: str, defines=()) -> str:
    """Compile ``body`` behind the step engine's header, run it, return what it printed."""
    src, exe = tmp_path / "case.cu", tmp_path / "case"
    src.write_text('#include "device/engine.h"\n#include <stdio.h>\n#include <string.h>\nusing namespace dfccl;\n' + body)
    cmd = [_build.nvcc(), "-std=c++17", "-O2", "-DDF_FAST_BUILD", *(f"-D{d}" for d in defines), "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(_build.CSRC / "src"),
           "-I", str(_build.CSRC / "include"), str(src), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.parametrize("skew", [0, 3])
def test_pieces_beyond_4_gib(tmp_path, skew):
    """A block's share of a pushed piece longer than 4 GiB: the first 4 GiB are one 64 MiB file mapped again and again, on either
    side, and a file of its own follows."""
    out = run_on_host(tmp_path, r"""
#include <sys/mman.h>
#include <unistd.h>
static const size_t CHUNK = 64u << 20, LEAD = 4ull << 30;
static char* area(int* first, int* last) {
  char* p = (char*)mmap(nullptr, LEAD + CHUNK, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  *first = memfd_create("first", 0); *last = memfd_create("last", 0);
  if (ftruncate(*first, CHUNK) || ftruncate(*last, CHUNK)) return nullptr;
  for (size_t o = 0; o < LEAD + CHUNK; o += CHUNK)
    if (mmap(p + o, CHUNK, PROT_READ | PROT_WRITE, MAP_SHARED | MAP_FIXED, o < LEAD ? *first : *last, 0) == MAP_FAILED) return nullptr;
  return p;
}
int main() {
  int f[4];
  char *src = area(f, f + 1), *dst = area(f + 2, f + 3);
  if (!src || !dst) return 2;
  const size_t tail = 1 << 20;
  memset(src, 1, CHUNK); memset(src + LEAD, 2, CHUNK);
  copyOne(src + SKEW, dst, LEAD + tail);
  for (size_t i = 0; i < CHUNK; ++i) if (dst[i] != (i < CHUNK - SKEW ? 1 : 2)) return 3;
  for (size_t i = 0; i < CHUNK; ++i) if (dst[LEAD + i] != (i < tail ? 2 : 0)) { printf("byte %zu behind 4 GiB: %d\n", i, dst[LEAD + i]); return 4; }
  puts("ok");
  return 0;
}
""".replace("SKEW", str(skew)))
    assert out == "ok\n"


def test_verdict_of_blocks_that_fail_for_different_causes(tmp_path):
    """A cause that a block reported, never one between two (1 timed out, 2 aborted, 3 bad argument): a bad argument before a wait
    that ran out before an abort, whatever the order; the word the blocks share is clear afterwards."""
    out = run_on_host(tmp_path, r"""
#include <memory>
#include <vector>
static int verdict(const std::vector<uint32_t>& status) {
  uint32_t done = 0;
  uint64_t flag = 0, ring[4] = {};
  RankDev rd;
  memset(&rd, 0, sizeof(rd));
  rd.doneCount = &done; rd.doneEpoch = &flag; rd.hostCq = ring; rd.cqCap = 4;
  std::unique_ptr<BlockShared> sh(new BlockShared);
  memset((void*)sh.get(), 0, sizeof(BlockShared));
  sh->k = rd;
  for (size_t b = 0; b < status.size(); ++b) {
    sh->cs.nBlocks = (int)status.size(); sh->loadedColl = 0; sh->dyn.epoch = 7; sh->dyn.status = status[b];
    completeColl(sh.get(), &rd, (int)b);
    if ((rd.devCqTail != 0) != (b + 1 == status.size())) return -1;
  }
  if (done != 0 || flag != ((uint64_t)cqeStatus(ring[0]) << 56 | 7)) return -2;
  return (int)cqeStatus(ring[0]);
}
int main() {
  for (auto& s : std::vector<std::vector<uint32_t>>{{0, 0}, {0, 1}, {2, 0, 0}, {3}, {1, 2}, {2, 1, 2, 2}, {1, 3}, {3, 1}, {2, 3, 2}, {1, 2, 3}}) printf("%d ", verdict(s));
  for (uint32_t s = 0; s < 4; ++s) printf("%d ", verdict(std::vector<uint32_t>(DF_MAX_BLOCKS, s)));
  return 0;
}
""")
    assert out.split() == "0 1 2 3 1 1 3 3 3 3 0 1 2 3".split()


def test_offsets_are_those_of_the_epoch(tmp_path):
    """Members on one device: whatever order the words of a slot arrive in, a wait succeeds with the offsets of its own epoch, also
    where the tag's 16 bits come round, and never with those of a peer that has gone on without it."""
    out = run_on_host(tmp_path, r"""
#include <memory>
static bool arrived(FlagSlot* f, uint32_t epoch, uint64_t* send, uint64_t* recv) {
  static DaemonCtl ctl;
  RankDev rd;
  memset((void*)&rd, 0, sizeof(rd));
  rd.ctl = &ctl;
  std::unique_ptr<BlockShared> sh(new BlockShared);
  memset((void*)sh.get(), 0, sizeof(BlockShared));
  sh->k = rd;
  CollStatic* c = &sh->cs;
  c->kind = dfcclCollBroadcast; c->inType = c->outType = ncclInt8; c->nranks = 2; c->root = 1; c->nBlocks = 1; c->count = 64;
  c->algo = dfcclAlgoOneShot; c->oneDevice = 1; c->myFlags = f; c->scale = 1.0;
  planColl(c, 0);
  sh->dyn.epoch = epoch;
  const bool ok = boundedWait(sh.get(), &rd, 0, 0, 4);
  *send = sh->peerSend[1]; *recv = sh->peerRecv[1];
  return ok;
}
int main() {
  for (uint32_t epoch : {1u, 2u, 0xffffu, 0x10000u, 0x10001u, 0x20000u, 0xffff0000u}) {
    for (int seen = 0; seen < 8; ++seen) {               // bit by bit: the arrival, the send offset, the receive offset are there
      FlagSlot f[2];
      memset((void*)f, 0, sizeof(f));
      f[1].arrive = seen & 1 ? epoch : epoch - 1;
      f[1].sendOff = seen & 2 ? offTagged(4096, epoch) : epoch > 1 ? offTagged(512, epoch - 1) : 0;
      f[1].recvOff = seen & 4 ? offTagged(8192, epoch) : epoch > 1 ? offTagged(1024, epoch - 1) : 0;
      uint64_t s, r;
      const bool ok = arrived(f, epoch, &s, &r);
      if (ok != (seen == 7)) { printf("epoch %u words %d: %d\n", epoch, seen, ok); return 1; }
      if (ok && (s != 4096 || r != 8192)) return 2;
      f[1].arrive = epoch + 1;                           // the peer has gone on
      f[1].sendOff = offTagged(512, epoch + 1);
      if (arrived(f, epoch, &s, &r)) return 3;
    }
  }
  puts("ok");
  return 0;
}
""")
    assert out == "ok\n"


def test_shifted_packs_are_made_once_each(tmp_path):
    """Warps of 32 lanes: every logical pack is made by one lane, whose neighbour has loaded the pack behind it; nothing is loaded
    beyond aligned pack nPacks; the lanes of a warp go round together."""
    out = run_on_host(tmp_path, r"""
#include <vector>
int main() {
  for (uint32_t nt : {32u, 64u, 480u})
    for (uint32_t unroll : {1u, 2u, 4u, 8u})
      for (uint64_t nPacks : {1ull, 2ull, 30ull, 31ull, 32ull, 62ull, 63ull, 464ull, 465ull, 466ull, 929ull, 930ull, 3719ull, 3720ull, 3721ull, 10007ull}) {
        std::vector<int> made(nPacks, 0);
        for (uint32_t warp = 0; warp < nt / 32; ++warp) {
          ShiftedWalk w[32];
          for (uint32_t l = 0; l < 32; ++l) w[l] = shiftedWalk(warp * 32 + l, nt, 32);
          for (uint64_t trip = 0;; ++trip) {
            const uint64_t hop = trip * unroll * w[0].step;
            const bool go = shiftedWarpAt(w[0].first + hop, w[0].lane, nPacks);
            for (uint32_t l = 0; l < 32; ++l) if (shiftedWarpAt(w[l].first + hop, w[l].lane, nPacks) != go) return 1;
            if (!go) break;
            for (uint32_t u = 0; u < unroll; ++u)
              for (uint32_t l = 0; l < 32; ++l) {
                const uint64_t q = w[l].first + hop + (uint64_t)u * w[l].step;
                if (w[l].lane != l || (shiftedLoads(q, l, nPacks) && q > nPacks)) return 2;
                if (!shiftedMakes(l, 32) || q >= nPacks) continue;
                if (!shiftedLoads(q, l, nPacks) || !shiftedLoads(q + 1, l + 1, nPacks) || w[l + 1].first != w[l].first + 1) return 3;
                ++made[q];
              }
          }
        }
        for (int m : made) if (m != 1) { printf("%u threads, %u, %llu packs: one made %d times\n", nt, unroll, (unsigned long long)nPacks, m); return 4; }
      }
  puts("ok");
  return 0;
}
""")
    assert out == "ok\n"


def test_shifted_sums_and_copies_stay_in_their_buffers(tmp_path):
    """Sums of one to nine sources and copies of pieces off the 16-byte grid, whose last wanted byte is the last of a page with nothing
    behind it and whose first is the first of one with nothing in front of it."""
    out = run_on_host(tmp_path, r"""
#include <sys/mman.h>
#include <vector>
#include <memory>
static const size_t PAGE = 4096, SPAN = 4 * PAGE;
static char* page() {                                  // SPAN bytes between two pages that cannot be touched
  char* p = (char*)mmap(nullptr, SPAN + 2 * PAGE, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  return mprotect(p + PAGE, SPAN, PROT_READ | PROT_WRITE) ? nullptr : p + PAGE;
}
int main() {
  std::unique_ptr<DataArgs> a(new DataArgs);
  std::vector<char*> in;
  for (int j = 0; j < 9; ++j) in.push_back(page());
  std::vector<char> out(SPAN + 128);
  for (int atEnd = 0; atEnd < 2; ++atEnd)
    for (int nsrc = 0; nsrc <= 9; ++nsrc)              // 0: a copy
      for (uint32_t bytes : {20u, 36u, 64u, 516u, 1028u, 2052u, 8188u, 16380u})
        for (uint32_t skew : {0u, 4u, 8u, 12u}) {      // of the destination, against sources whose ends or beginnings lie on the grid
          const uint32_t n = bytes / 4;
          memset((void*)a.get(), 0, sizeof(DataArgs));
          char* dst = (char*)(((uintptr_t)out.data() + 32) & ~(uintptr_t)31) + 32 + skew;
          memset(out.data(), 7, out.size());
          const size_t at = atEnd ? SPAN - bytes : 0;
          for (int j = 0; j < (nsrc ? nsrc : 1); ++j) {
            a->src[j] = in[j] + at;
            for (uint32_t i = 0; i < n; ++i) ((float*)a->src[j])[i] = (float)((i * 37 + j * 101) % 1009) + 0.25f * j;
          }
          a->dst[0] = dst; a->nsrc = nsrc ? nsrc : 1; a->ndst = 1; a->scale = 1.0; a->postDiv = 0;
          if (nsrc) { a->n = n; if (!reduce_dispatch(ncclFloat32, ncclFloat32, OP_SUM, a.get())) return 2; }
          else { a->n = bytes; copy_multi(a.get()); }
          for (uint32_t i = 0; i < n; ++i) {
            float s = ((const float*)a->src[0])[i];
            for (int j = 1; j < nsrc; ++j) s += ((const float*)a->src[j])[i];
            if (((const float*)dst)[i] != s) { printf("%d sources, %u bytes, skew %u: element %u\n", nsrc, bytes, skew, i); return 3; }
          }
          if (dst[-1] != 7 || dst[bytes] != 7) return 4;
        }
  puts("ok");
  return 0;
}
""", defines=("DF_DATAPATH_IMPL",))
    assert out == "ok\n"


def test_an_entry_that_cannot_be_taken_ends_no_wait(tmp_path):
    """The next submission of a collective that still runs stays at the head of the ring: the wait that has nothing else to do keeps its
    budget; an entry that can be taken ends it at the fourth poll (at the sixteenth where the peers have arrived), one that a stream
    has yet to release at the twentieth (thirty-second)."""
    out = run_on_host(tmp_path, r"""
#include "device/daemon_impl.h"
#include <memory>
static DaemonCtl ctl;
static RankDev rd;
static SqSlot ring[8];
static FlagSlot flags[2];
static uint32_t meta[4];
static CollDyn dyn[4];
static uint64_t frontier;
static std::unique_ptr<BlockShared> sh;
static void put(uint64_t index, int coll, uint32_t flags = 0) {
  Sqe q;
  memset((void*)&q, 0, sizeof(q));
  q.collId = coll; q.epoch = 2; q.flags = flags;
  ring[index & 7] = sqEncode(q, sqTag(index, 8));
}
static void say(int v) { printf("%d ", v); }
static int take() {
  SqSlot slot, next;
  const bool haveNext = sqPeek(&sh->k, sh->frontier + 1, &next), have = sqPeek(&sh->k, sh->frontier, &slot);
  return have ? consumeSubmissions(sh.get(), &rd, 0, slot, next, haveNext) : 0;
}
static int polls(int which) {
  if (boundedWait(sh.get(), &rd, 0, which, 200)) return -1;
  return (int)sh->waitSpins;
}
int main() {
  memset((void*)&rd, 0, sizeof(rd)); memset((void*)ring, 0, sizeof(ring));
  rd.ctl = &ctl; rd.spinBudget = 32; rd.headTries = 5; rd.devSq = ring; rd.sqCap = 8; rd.nBlocks = 1; rd.maxColls = 4; rd.meta = meta; rd.dyn = dyn; rd.hostFrontier = &frontier;
  for (auto& m : meta) m = DF_META_VALID | 1u;
  sh.reset(new BlockShared);
  memset((void*)sh.get(), 0, sizeof(BlockShared));
  BlockSaved sv;
  memset((void*)&sv, 0, sizeof(sv));
  rd.saved = &sv;
  blockRestore(sh.get(), &rd, 0);
  CollStatic* c = &sh->cs;
  c->kind = dfcclCollBroadcast; c->inType = c->outType = ncclInt8; c->nranks = 2; c->root = 1; c->nBlocks = 1; c->count = 64;
  c->algo = dfcclAlgoOneShot; c->oneDevice = 1; c->myFlags = flags; c->scale = 1.0;
  planColl(c, 0);
  put(0, 1);
  say(take());                                         // collective 1 runs, its peer is not there
  sh->dyn.epoch = 2;
  say(polls(0)); say(polls(1));
  put(1, 1);                                           // its next submission: stays where it is
  say(polls(0)); say(take());                          // (the wait that meets it first ends)
  say(polls(0)); say(polls(1));
  sh->busy[0] = 0;                                     // collective 1 has completed
  say(take());
  put(2, 2);
  say(polls(0)); say(polls(1)); say(take()); say(polls(0));
  put(3, 3, SQE_TRIGGERED);                            // a stream has yet to release it
  say(polls(0)); say(polls(1)); say(take()); say((int)sh->nTrig);
  return 0;
}
""")
    assert out.split() == "1 200 200 4 0 200 200 1 4 16 1 200 20 32 1 1".split()


def test_how_long_a_wait_lasts(tmp_path):
    """RECV_SUCCESS_FACTOR: a wait that succeeded at its first poll allows the next of the same submission `factor` polls, where that is
    more than its budget and nothing else is queued or may be released.  NUM_TRY_TASKQ_HEAD: beside others the oldest of the queue has
    that many budgets where a stream released it."""
    out = run_on_host(tmp_path, r"""
#include <memory>
static DaemonCtl ctl;
static uint32_t polls(uint32_t factor, uint32_t budget, uint32_t queued, uint32_t waiting = 0, uint32_t flags = 0, int place = 0) {
  FlagSlot f[2];
  memset((void*)f, 0, sizeof(f));
  RankDev rd;
  memset((void*)&rd, 0, sizeof(rd));
  rd.ctl = &ctl; rd.recvSuccessFactor = factor; rd.spinBudget = 32; rd.headTries = 5;
  std::unique_ptr<BlockShared> sh(new BlockShared);
  memset((void*)sh.get(), 0, sizeof(BlockShared));
  sh->k = rd; sh->nActive = queued; sh->nTrig = waiting; sh->loadedColl = 3;
  for (uint32_t i = 0; i < queued; ++i) sh->active[i] = (int)i == place ? 3 : 7;
  CollStatic* c = &sh->cs;
  c->kind = dfcclCollBroadcast; c->inType = c->outType = ncclInt8; c->nranks = 2; c->root = 1; c->nBlocks = 1; c->count = 64;
  c->algo = dfcclAlgoOneShot; c->oneDevice = 1; c->myFlags = f; c->scale = 1.0;
  planColl(c, 0);
  sh->dyn.epoch = 1; sh->dyn.sqeFlags = flags;
  f[1].arrive = 1; f[1].sendOff = offTagged(64, 1); f[1].recvOff = offTagged(128, 1);
  if (!patientWait(sh.get(), &rd, 0, 0, budget) || sh->waitSpins != 1) return 0;
  if (patientWait(sh.get(), &rd, 0, 1, budget)) return 1;      // the peer is never done
  return sh->waitSpins;
}
int main() {
  printf("%u %u %u %u %u ", polls(0, 2, 1), polls(50, 2, 1), polls(50, 160, 1), polls(50, 2, 2), polls(1u << 30, 2, 1));
  printf("%u %u %u %u %u\n", polls(50, 20, 1, 1), polls(0, 2, 2, 0, SQE_TRIGGERED), polls(0, 2, 2, 0, SQE_TRIGGERED, 1), polls(50, 2, 2, 3, SQE_TRIGGERED), polls(0, 160, 1, 0, SQE_TRIGGERED));
  return 0;
}
""")
    assert out.split() == ["2", "50", "160", "2", str(64 * 32), "20", "10", "2", "10", "160"]
