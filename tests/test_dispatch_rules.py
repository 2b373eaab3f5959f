"""Which kernel a size takes, as far as that can be asked without a GPU (148 SMs)."""
import pytest

from dfccl_b200 import native as nv


@pytest.mark.parametrize("rows,n", [(16384, 8), (16384, 256), (24576, 1024), (65536, 64), (65536, 256), (131072, 1984)])
def test_tall_column_sums_fill_the_gpu(rows, n):
    """Blocks of 64 columns and a stretch of at least 128 rows each: as many as the GPU has SMs."""
    words = nv.lib().dfcclColumnSumWork(rows, n)
    assert words % n == 0
    stretches = words // n
    assert stretches * ((n + 63) // 64) >= min(148, rows // 128) and stretches <= rows // 128


@pytest.mark.parametrize("rows,n", [(1, 8), (8192, 1024), (16383, 64), (65536, 2048), (131072, 4096)])
def test_other_column_sums_are_one_launch(rows, n):
    assert nv.lib().dfcclColumnSumWork(rows, n) == 0


def gemm_plan(m, n, k, b_transposed=False, epilogue=0, sms=148):
    """(pairs, tile columns, slices, width of a persistent tile)"""
    import ctypes as C
    plan = (C.c_int * 4)()
    nv.check(nv.lib().dfcclGemmPlan(m, n, k, int(b_transposed), epilogue, sms, plan), "dfcclGemmPlan")
    return tuple(plan)


@pytest.mark.parametrize("m,n,k", [(4096, 1024, 8192), (1024, 4096, 8192), (4096, 1024, 1024), (2304, 2048, 8192), (9472, 512, 8192)])
def test_one_wave_of_the_widest_tiles(m, n, k):
    """Plain products of at most a tile per pair of SMs run on the tile kernel, whatever the storage order; with an epilogue, with
    more tiles than pairs, with a short contraction or less than three row tiles on the persistent one."""
    for bt in (False, True):
        assert gemm_plan(m, n, k, bt) == (1, 256, 1, 0)
    assert gemm_plan(m, n, k, False, 1)[3] == 256
    assert gemm_plan(2 * m, n, k)[3] == gemm_plan(2 * m, n, k, True)[3] == 256
    assert gemm_plan(m, n, 448)[1] != 256 and gemm_plan(512, 7168, k)[1] != 256


def test_widths_of_the_persistent_kernel():
    """What its tiles can be: 64 columns and more, 128 and more where B is stored MN-major (what its tests run is all of it)."""
    seen = {bt: {gemm_plan(128 * m, 256 * n, 64 * k, bt, e)[3] for m in range(1, 33) for n in range(1, 33) for k in (1, 2, 3, 5, 8, 16, 36, 60, 128) for e in (0, 1)}
            for bt in (False, True)}
    assert seen[False] - {0} == {64, 96, 128, 160, 192, 224, 256} and seen[True] - {0} == {128, 160, 192, 224, 256}
