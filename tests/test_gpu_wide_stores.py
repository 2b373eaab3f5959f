"""bf16 / fp16 -> fp32 collectives write 32 bytes per thread: outputs on 32-byte boundaries, on 16-byte ones and on neither."""
import pytest
import torch

from helpers import run_ranks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ranks", [1, 3])
@pytest.mark.parametrize("out_off", [0, 4, 8, 5])                      # fp32 elements: 0, 16, 32 and 20 bytes
def test_half_to_float_outputs(native, ranks, out_off):
    from dfccl_b200.utils import tensor_from_ptr
    native.set_backend("cuda")
    torch.cuda.set_device(0)
    comms = native.Comm.init_loopback(ranks, 0)
    counts = [7, 8, 4099, 300000]
    bad = []

    def body(r):
        ctx = native.RankCtx(r, 0)
        ctx.set_daemon_geometry(4, 0)
        for i, n in enumerate(counts):
            ctx.prepare(i, comms[r], native.ALLREDUCE, n, native.BFLOAT16, out_dtype=native.FLOAT32, scale=0.5)
        ctx.finalize()
        st = torch.cuda.Stream()
        for i, n in enumerate(counts):
            p, q = comms[r].alloc(2 * n), comms[r].alloc(4 * (n + 32))
            x, y = tensor_from_ptr(p, (n,), torch.bfloat16, "cuda:0"), tensor_from_ptr(q, (n + 32,), torch.float32, "cuda:0")
            x.copy_((torch.arange(n, device="cuda") % 251 + r).to(torch.bfloat16))
            y.fill_(-1.0)
            torch.cuda.current_stream().synchronize()
            if ranks == 1:
                ctx.run_on_stream(i, p, q + 4 * out_off, st.cuda_stream)
            else:
                ctx.run(i, p, q + 4 * out_off)
            assert ctx.wait(i, 60000) == native.SUCCESS
            want = sum(((torch.arange(n, device="cuda") % 251 + k).to(torch.bfloat16).float() for k in range(ranks))) * 0.5
            if not (torch.equal(y[out_off:out_off + n], want) and bool((y[:out_off] == -1).all()) and bool((y[out_off + n:] == -1).all())):
                bad.append((r, n))
        ctx.destroy()

    run_ranks(ranks, body, timeout=120)
    for c in comms:
        c.destroy()
    assert not bad


@pytest.mark.parametrize("ranks", [2, 5, 8])
def test_short_calls_of_many_sources(native, ranks):
    """Calls of less than a trip of the block (four sources at a time, the ragged end on the warps the packs leave idle):
    around whole packs, warps and the block's threads, aligned or not."""
    from dfccl_b200.utils import tensor_from_ptr
    native.set_backend("cuda")
    torch.cuda.set_device(0)
    comms = native.Comm.init_loopback(ranks, 0)
    counts = [1, 5, 8, 63, 248, 255, 256, 509, 3839, 4097, 16403]
    bad = []

    def body(r):
        ctx = native.RankCtx(r, 0)
        ctx.set_daemon_geometry(2, 0)
        for i, n in enumerate(counts):
            ctx.prepare(2 * i, comms[r], native.ALLREDUCE, n, native.FLOAT16)
            ctx.prepare(2 * i + 1, comms[r], native.REDUCESCATTER, n, native.INT32, op=native.MAX)
        ctx.finalize()
        for i, n in enumerate(counts):
            value = lambda k, m: (torch.arange(m, device="cuda") * 7 + 13 * k) % 101                  # noqa: E731
            p, q = comms[r].alloc(2 * n + 64), comms[r].alloc(2 * n + 64)
            x, y = (tensor_from_ptr(a + 6, (n,), torch.float16, "cuda:0") for a in (p, q))            # off the 16-byte grid alike
            s, d = comms[r].alloc(4 * n * ranks), comms[r].alloc(4 * n)
            u, v = tensor_from_ptr(s, (n * ranks,), torch.int32, "cuda:0"), tensor_from_ptr(d, (n,), torch.int32, "cuda:0")
            x.copy_(value(r, n).to(torch.float16))
            u.copy_(value(r, n * ranks).to(torch.int32))
            y.zero_(), v.zero_()
            torch.cuda.current_stream().synchronize()
            ctx.run(2 * i, p + 6, q + 6)
            ctx.run(2 * i + 1, s, d)
            assert ctx.wait_all(60000) == native.SUCCESS
            want = sum(value(k, n) for k in range(ranks)).to(torch.float16)                           # whole numbers below 2048: exact
            top = torch.stack([value(k, n * ranks) for k in range(ranks)]).amax(0).to(torch.int32)[r * n:(r + 1) * n]
            if not (torch.equal(y, want) and torch.equal(v, top)):
                bad.append((r, n))
        ctx.destroy()

    run_ranks(ranks, body, timeout=120)
    for c in comms:
        c.destroy()
    assert not bad
