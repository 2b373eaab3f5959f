"""Long sums of two, four and eight aligned sources, whose loads run ahead of the stores: whole trips of a block, one pack more and
less, ragged ends (all-reduces: the pieces of a reduce-scatter of odd length start off the grid), every element size, results wider and
narrower than the operands, in place and not; and sums and copies of pieces that start off the 16-byte grid, where a warp's 32
aligned packs make 31."""
import pytest

from test_gpu_daemon import TORCH_OF, _loopback_case, nv  # noqa: F401

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
        pack = 16 // TORCH_OF[dtype].itemsize
        count = (count + pack - 1) // pack * pack          # chunks on the 16-byte grid; others take the shifted path
    _loopback_case(nv, kind, nranks, count, dtype, op=op, out_name=out, blocks=1)


# 465 packs of 16 bytes are what a block's 15 warps make of one load each
SHIFTED = [("reducescatter", 2, 4 * 465 * 40 + 1, "FLOAT32", None), ("reducescatter", 4, 4 * 465 * 38 + 3, "FLOAT32", None), ("reducescatter", 4, 4 * 465 + 3, "FLOAT32", None),
           ("reducescatter", 8, 8 * 465 * 36 + 1, "BFLOAT16", None), ("reducescatter", 4, 8 * 465 * 37 - 3, "BFLOAT16", "FLOAT32"), ("reducescatter", 3, 4 * 465 * 40 + 3, "FLOAT32", None),
           ("reducescatter", 2, 4 * 465 * 41 - 1, "FLOAT32", "BFLOAT16"), ("reducescatter", 8, 8 * 465 * 35 + 9, "FLOAT16", "FLOAT32"), ("reducescatter", 4, 16 * 465 * 36 + 5, "UINT8", None),
           ("allgather", 4, 8 * 465 * 40 + 7, "BFLOAT16", None), ("allgather", 2, 16 * 465 * 8 * 5 + 3, "UINT8", None), ("allgather", 2, 4 * 465 * 8 * 5 + 1, "FLOAT32", None), ("allgather", 8, 8 * 31 + 5, "BFLOAT16", None)]


@pytest.mark.parametrize("kind,nranks,count,dtype,out", SHIFTED)
def test_pieces_off_the_grid(nv, kind, nranks, count, dtype, out):  # noqa: F811
    for blocks in (1, 3):
        _loopback_case(nv, kind, nranks, count, dtype, out_name=out, blocks=blocks)


# every source's next packs are loaded in front of the present ones' stores, which go to one of the sources
IN_PLACE = [("allreduce", 2, 8 * 1920 * 7 + 5, "BFLOAT16", "SUM"), ("allreduce", 4, 4 * 960 * 4 * 5 + 3, "FLOAT32", "AVG"), ("allreduce", 8, 8 * 480 * 8 * 5 + 1, "BFLOAT16", "SUM"),
            ("allreduce", 4, 300007, "INT32", "MAX"), ("reducescatter", 2, 4 * 1920 * 9 + 4, "FLOAT32", "SUM"), ("reducescatter", 4, 8 * 960 * 5 - 8, "BFLOAT16", "SUM"),
            ("reducescatter", 8, 4 * 480 * 40 + 3, "FLOAT32", "SUM"), ("allgather", 4, 300007, "BFLOAT16", "SUM")]


@pytest.mark.parametrize("kind,nranks,count,dtype,op", IN_PLACE)
def test_long_calls_in_place(nv, kind, nranks, count, dtype, op):  # noqa: F811
    for blocks in (1, 3):
        _loopback_case(nv, kind, nranks, count, dtype, op=op, in_place=True, iters=3, blocks=blocks, algo=nv.ALGO_TWOSHOT if kind == "allreduce" else 0)
