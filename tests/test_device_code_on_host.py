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
