"""Long sums of two, four and eight aligned sources, whose loads run ahead of the stores: whole trips of a block, one pack more and
less, ragged ends, every element size, results wider and narrower than the operands."""
import pytest

from test_gpu_daemon import _loopback_case, nv  # noqa: F401

pytestmark = pytest.mark.gpu

# a block of 480 threads takes 1920 packs of 16 bytes a trip among two ranks, 960 among four (480 where the result is twice as wide), 480 among eight
CASES = [(2, 4 * 1920 * 3, "FLOAT32", None, "AVG"), (2, 8 * 1920 * 4 + 8, "BFLOAT16", None, "SUM"), (2, 8 * 1920 * 3 - 8, "BFLOAT16", "FLOAT32", "SUM"),
         (2, 8 * 1920 * 5 + 8 * 479 + 5, "FLOAT16", None, "SUM"), (4, 4 * 960 * 7, "INT32", None, "AVG"), (4, 8 * 480 * 11 + 3, "BFLOAT16", "FLOAT32", "SUM"),
         (4, 4 * 960 * 9 - 4, "FLOAT32", "BFLOAT16", "SUM"), (4, 2 * 960 * 6 + 1, "FLOAT64", None, "SUM"), (8, 8 * 480 * 7 + 8, "BFLOAT16", None, "SUM"),
         (8, 16 * 480 * 6 - 1, "UINT8", None, "SUM"), (8, 700003, "FLOAT32", None, "SUM"), (8, 8 * 480 * 9 + 7, "FLOAT16", "FLOAT32", "SUM")]


@pytest.mark.parametrize("kind", ["allreduce", "reducescatter"])
@pytest.mark.parametrize("nranks,count,dtype,out,op", CASES)
def test_sums_with_loads_ahead(nv, kind, nranks, count, dtype, out, op):  # noqa: F811
    if kind == "reducescatter":
        count = (count + 15) // 16 * 16                    # chunks on the 16-byte grid; others take the shifted path
    _loopback_case(nv, kind, nranks, count, dtype, op=op, out_name=out, blocks=1)
