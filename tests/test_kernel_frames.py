"""What the out-of-line bodies of the data path save of their caller's registers, as the compiler reports it."""
import re
import subprocess

from dfccl_b200 import _build


def test_calls_on_the_grid_do_not_pay_for_shifting(tmp_path):
    """Bytes of frame of the bodies for maxima, minima and products, and of copies, on the 16-byte grid: no more than they had while
    shifted sources, in the same body, kept one load in flight (112 bf16, 120 fp32, 112 copies)."""
    cmd = [_build.nvcc(), "-std=c++17", "-O3", "-lineinfo", "-DDF_FAST_BUILD", "-rdc=true", *_build.ARCH, "-maxrregcount=128", "-Xptxas", "-v",
           "-I", str(_build.CSRC / "include"), "-c", str(_build.CSRC / "src/device/datapath.cu"), "-o", str(tmp_path / "datapath.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    frames = {name: int(size) for name, size in re.findall(r"Function properties for (\S+)\s+(\d+) bytes stack frame", r.stderr)}
    grid = {n: s for n, s in frames.items() if re.search(r"reduceBody\S+Li[123]ELb0E", n)}
    assert len(grid) == 6 and max(grid.values()) <= 112, grid
    copies = {n: s for n, s in frames.items() if re.search(r"copy_on_grid", n)}
    assert len(copies) == 1 and max(copies.values()) <= 112, copies
