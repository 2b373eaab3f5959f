"""Parts of the device code compiled for the host by themselves, where the sizes or states they are about cannot be reached through
a communicator on this machine."""
import subprocess

import pytest

from dfccl_b200 import _build


def run_on_host(tmp_path, body: str) -> str:
    """Compile ``body`` behind the step engine's header, run it, return what it printed."""
    src, exe = tmp_path / "case.cu", tmp_path / "case"
    src.write_text('#include "device/engine.h"\n#include <stdio.h>\n#include <string.h>\nusing namespace dfccl;\n' + body)
    cmd = [_build.nvcc(), "-std=c++17", "-O2", "-DDF_FAST_BUILD", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(_build.CSRC / "src"),
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
