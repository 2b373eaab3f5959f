"""Small calls have bodies of their own on the device: sizes around one pack per thread, around the last size that takes them (four
packs of 16 bytes for each of the 480 working threads of a block), more sources than are loaded at a time, every operator."""
import pytest

from test_gpu_daemon import _loopback_case, nv  # noqa: F401

pytestmark = pytest.mark.gpu

LIMIT = 4 * 480 * 16


@pytest.mark.parametrize("dt,out,op,count", [
    ("BFLOAT16", "FLOAT32", "SUM", LIMIT // 2), ("BFLOAT16", "FLOAT32", "SUM", LIMIT // 2 + 1),
    ("BFLOAT16", "BFLOAT16", "SUM", 480 * 8), ("BFLOAT16", "BFLOAT16", "SUM", 480 * 8 + 7),
    ("FLOAT32", "BFLOAT16", "SUM", LIMIT // 4 - 1), ("FLOAT16", "FLOAT16", "AVG", 1001),
    ("INT8", "INT8", "MAX", LIMIT), ("INT8", "INT8", "MAX", LIMIT + 1), ("UINT8", "UINT8", "MIN", 15),
    ("FLOAT64", "FLOAT64", "PROD", LIMIT // 8 + 1), ("INT64", "INT64", "SUM", 479), ("INT32", "INT32", "SUM", LIMIT // 4)])
@pytest.mark.parametrize("nranks", [2, 7])
def test_small_all_reduce(nv, nranks, dt, out, op, count):  # noqa: F811
    _loopback_case(nv, "allreduce", nranks, count, dt, out_name=out, op=op)


@pytest.mark.parametrize("kind", ["allgather", "reducescatter", "broadcast"])
@pytest.mark.parametrize("dt,count,skew", [("BFLOAT16", LIMIT // 2 + 3, (0, 0)), ("FLOAT32", 481 * 4 + 1, (0, 0)), ("INT8", LIMIT + 17, (1, 6)),
                                           ("FLOAT32", 65539, (1, 0))])
def test_small_pieces(nv, kind, dt, count, skew):  # noqa: F811
    """Pieces of odd length lie off the 16-byte grid in the gathered and scattered arrays."""
    _loopback_case(nv, kind, 4, count, dt, skew=skew)
