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
