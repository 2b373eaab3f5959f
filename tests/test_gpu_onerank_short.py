"""Registered collectives of a one-rank job at the edges of the one-cluster form (8192 packs of 16 source bytes) and behind one
another in a stream, where the blocks of a call come up while the one in front still runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,out,count", [("BFLOAT16", "FLOAT32", 65536), ("BFLOAT16", "FLOAT32", 65537), ("BFLOAT16", "FLOAT32", 65544),
                                          ("FLOAT32", "FLOAT32", 32768), ("FLOAT32", "FLOAT32", 32771), ("FLOAT32", "FLOAT32", 3), ("INT8", "INT8", 131072 + 16)])
@pytest.mark.parametrize("skew", [0, 1])
def test_chain_of_short_calls(dt, out, count, skew):
    """Every call reads what the one in front has written; results and completions as of separate calls."""
    from dfccl_b200 import native as nv
    from dfccl_b200.utils.tensors import tensor_from_ptr
    nv.set_backend("cuda")
    torch.cuda.set_device(0)
    td, to = {"BFLOAT16": torch.bfloat16, "FLOAT32": torch.float32, "INT8": torch.int8}[dt], {"FLOAT32": torch.float32, "INT8": torch.int8}[out]
    (comm,) = nv.Comm.init_loopback(1, 0)
    ctx = nv.RankCtx(0, 0)
    scale = 1.0 if dt == "INT8" else 0.5
    ctx.prepare(0, comm, nv.ALLREDUCE, count, getattr(nv, dt), out_dtype=getattr(nv, out), scale=scale)
    for i in range(1, 6):
        ctx.prepare(i, comm, nv.ALLREDUCE, count, getattr(nv, out), scale=scale)
    ctx.finalize()
    es, eo = torch.empty((), dtype=td).element_size(), torch.empty((), dtype=to).element_size()
    ptrs = [comm.alloc(count * es + 64) + skew * es] + [comm.alloc(count * eo + 64) + skew * eo for _ in range(6)]
    bufs = [tensor_from_ptr(ptrs[0], (count,), td, "cuda:0")] + [tensor_from_ptr(p, (count,), to, "cuda:0") for p in ptrs[1:]]
    s = torch.cuda.current_stream().cuda_stream
    for it in range(3):
        x = torch.randint(-100, 101, (count,), device="cuda").to(td)
        bufs[0].copy_(x)
        for i in range(6):
            ctx.run_on_stream(i, ptrs[i], ptrs[i + 1], s)
        for i in range(6):
            ctx.stream_wait(i, s)
        want = x.to(to) if dt == "INT8" else x.to(to) * 0.5 ** 6
        assert torch.equal(bufs[6], want)                # powers of two: exact
    assert ctx.wait_all(30000) == nv.SUCCESS
    ctx.destroy()
    comm.destroy()
