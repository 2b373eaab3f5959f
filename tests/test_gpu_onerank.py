"""Collectives of a one-rank communicator run as one streaming kernel over the whole GPU (csrc/src/daemon/onerank.cu):
sizes around its pack, block and grid boundaries, buffers off the 16-byte grid, every element size."""
import ctypes as C
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

PACKS_OF_FOUR = 148 * 256 * 4           # 16-byte packs from which a thread takes four (148 SMs)


@pytest.fixture(scope="module")
def comm():
    from dfccl_b200 import native as nv
    nv.set_backend("cuda")
    torch.cuda.set_device(0)
    (c,) = nv.Comm.init_loopback(1, 0)
    yield c
    c.destroy()


@pytest.mark.parametrize("dt", ["float32", "bfloat16", "float16", "float64", "int32", "int8"])
@pytest.mark.parametrize("nbytes", [8, 16, 4096 - 8, 256 * 16 + 8, PACKS_OF_FOUR * 16 - 24, PACKS_OF_FOUR * 16 + 40])
@pytest.mark.parametrize("skew", [(0, 0), (1, 1), (1, 0)])
def test_premultiplied_sum_and_copies_of_one_rank(comm, dt, nbytes, skew):
    """A pre-multiplied sum is one multiplication in the accumulator type and one rounding: the result is exactly that
    of the same multiplication in PyTorch.  Kinds that only copy, and a plain sum in place, leave the bytes as they are."""
    from dfccl_b200 import native as nv
    from dfccl_b200.ops import collectives
    from dfccl_b200.utils import nccl_dtype
    tdt = getattr(torch, dt)
    n = nbytes // torch.empty((), dtype=tdt).element_size()
    g = torch.Generator(device="cuda").manual_seed(n)
    x = (torch.randn(n + 8, device="cuda", generator=g) * 50).to(tdt)[skew[0]:skew[0] + n]
    y = torch.zeros(n + 8, device="cuda", dtype=tdt)
    out = y[skew[1]:skew[1] + n]
    assert torch.equal(collectives.all_gather(comm, x, out), x)
    assert torch.equal(y[skew[1] + n:], torch.zeros_like(y[skew[1] + n:]))          # nothing behind the end
    z = x.clone()
    assert torch.equal(collectives.all_reduce(comm, z, op="avg"), x)
    if not tdt.is_floating_point:
        return
    L, op, s = nv.lib(), C.c_int(), C.c_float(0.3)
    nv.check(L.ncclRedOpCreatePreMulSum(C.byref(op), C.byref(s), nv.FLOAT32, 1, comm.handle))
    st = torch.cuda.current_stream().cuda_stream
    nv.check(L.ncclReduceScatter(x.data_ptr(), out.data_ptr(), n, nccl_dtype(tdt), op.value, comm.handle, st))
    nv.check(L.ncclRedOpDestroy(op.value, comm.handle))
    acc = torch.float64 if tdt == torch.float64 else torch.float32
    assert torch.equal(out, (x.to(acc) * torch.tensor(s.value, dtype=acc, device="cuda")).to(tdt))


@pytest.mark.parametrize("n", [1, 1000003])
@pytest.mark.parametrize("in_place", [False, True])
def test_registered_collective_of_one_rank_in_the_stream_and_through_the_daemon(n, in_place):
    """A stream-ordered submission of a one-rank collective runs in the stream itself; deferred and host submissions of
    the same id go through the daemon.  Mixed, they must count alike: a wait on another stream sees the right one, and
    every submission is delivered to the host."""
    from dfccl_b200 import native as nv
    from dfccl_b200.utils import tensor_from_ptr
    nv.set_backend("cuda")
    torch.cuda.set_device(0)
    (c,) = nv.Comm.init_loopback(1, 0)
    ctx = nv.RankCtx(0, 0)
    scale = 1.0 if in_place else 3.0
    ctx.prepare(0, c, nv.ALLREDUCE, n, nv.FLOAT32, scale=scale)
    ctx.finalize()
    p = c.alloc(4 * n)
    q = p if in_place else c.alloc(4 * n)
    x, y = tensor_from_ptr(p, (n,), torch.float32, "cuda:0"), tensor_from_ptr(q, (n,), torch.float32, "cuda:0")
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    for it in range(6):
        how = ("stream", "deferred", "host")[it % 3]
        with torch.cuda.stream(s1):
            x.fill_(float(it + 1))
            if how == "stream":
                ctx.run_on_stream(0, p, q, s1.cuda_stream)
            elif how == "deferred":
                ctx.run_deferred(0, p, q)
                ctx.trigger_on_stream(0, s1.cuda_stream)
            else:
                s1.synchronize()
                ctx.run(0, p, q)
            ctx.stream_wait(0, s1.cuda_stream)
            a = y.sum(dtype=torch.float64)
        with torch.cuda.stream(s2):
            ctx.stream_wait(0, s2.cuda_stream)
            b = y.sum(dtype=torch.float64)
        torch.cuda.synchronize()
        assert float(a) == float(b) == scale * (it + 1) * n, (it, how)
    assert ctx.wait_all(10000) == nv.SUCCESS
    st = ctx.stats()
    assert st["sqesSubmitted"] == st["cqesDelivered"] == 6
    ctx.destroy()
    c.destroy()


def test_abort_waits_for_a_collective_that_is_being_launched():
    """The launch queue of a stream holds about a thousand kernels: a thread that goes on calling behind a long kernel ends up
    waiting inside a call.  An abort by another thread returns only after that call has left the communicator."""
    from dfccl_b200 import native as nv
    nv.set_backend("cuda")
    torch.cuda.set_device(0)
    (c,) = nv.Comm.init_loopback(1, 0)
    x, y = torch.ones(64, device="cuda"), torch.empty(64, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(2_000_000_000)                       # about a second
    state = {"inside": 0.0, "stop": False, "left": 0.0}

    def caller():
        torch.cuda.set_device(0)
        while not state["stop"]:
            state["inside"] = time.perf_counter()
            assert nv.lib().ncclAllReduce(x.data_ptr(), y.data_ptr(), 64, nv.FLOAT32, nv.SUM, c.handle, s.cuda_stream) == nv.SUCCESS
            state["inside"] = 0.0
        state["left"] = time.perf_counter()

    t = threading.Thread(target=caller)
    t.start()
    deadline = time.perf_counter() + 5
    while time.perf_counter() < deadline and not (state["inside"] and time.perf_counter() - state["inside"] > 0.1):
        time.sleep(0.001)
    stuck = bool(state["inside"])
    state["stop"] = True
    if not stuck:                                              # (a deeper queue: nothing to see)
        t.join()
        c.destroy()
        pytest.skip("no call came to wait for the launch queue")
    c._live = False
    r = nv.lib().ncclCommAbort(c.handle)
    after = time.perf_counter()
    t.join(30)
    assert r == nv.SUCCESS and state["left"] and state["left"] - after < 0.05
    torch.cuda.synchronize()
    assert torch.equal(x, y)


def test_a_captured_wait_orders_its_graph_behind_an_earlier_collective():
    """The collective ran in the stream that is then captured; the graph is replayed on another one."""
    from dfccl_b200 import native as nv
    from dfccl_b200.utils import tensor_from_ptr
    nv.set_backend("cuda")
    torch.cuda.set_device(0)
    (c,) = nv.Comm.init_loopback(1, 0)
    n = 1 << 20
    ctx = nv.RankCtx(0, 0)
    ctx.prepare(0, c, nv.ALLREDUCE, n, nv.FLOAT32, scale=2.0)
    ctx.finalize()
    p, q = c.alloc(4 * n), c.alloc(4 * n)
    x, y = tensor_from_ptr(p, (n,), torch.float32, "cuda:0"), tensor_from_ptr(q, (n,), torch.float32, "cuda:0")
    seen = torch.zeros(n, device="cuda")
    x.fill_(1.0)
    y.zero_()
    torch.cuda.synchronize()
    s, other, g = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        torch.cuda._sleep(400_000_000)                          # about 0.2 s: the capture is over and replayed before the collective
        ctx.run_on_stream(0, p, q, s.cuda_stream)
        g.capture_begin(capture_error_mode="thread_local")      # (the library's own threads go on calling the runtime)
        try:
            ctx.stream_wait(0, s.cuda_stream)
            seen.copy_(y)
        finally:
            g.capture_end()
    with torch.cuda.stream(other):
        g.replay()
    torch.cuda.synchronize()
    assert bool((seen == 2.0).all())
    assert ctx.wait_all(10000) == nv.SUCCESS
    ctx.destroy()
    c.destroy()


@pytest.mark.parametrize("kind,reduced,copied", [("ALLREDUCE", 1, 0), ("REDUCESCATTER", 1, 0), ("ALLGATHER", 0, 1), ("BROADCAST", 0, 1)])
def test_collectives_in_the_stream_are_counted_and_traced(kind, reduced, copied, tmp_path, monkeypatch):
    """As the daemon's are: bytes in the statistics, the events of a collective's life in the trace."""
    import json
    from dfccl_b200 import native as nv
    nv.set_backend("cuda")
    torch.cuda.set_device(0)
    monkeypatch.setenv("DFCCL_TRACE", "1")
    (c,) = nv.Comm.init_loopback(1, 0)
    n, calls = 3001, 3
    ctx = nv.RankCtx(0, 0)
    ctx.prepare(7, c, getattr(nv, kind), n, nv.FLOAT32)
    ctx.finalize()
    x, y = torch.randn(n, device="cuda"), torch.zeros(n, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for _ in range(calls):
        ctx.run_on_stream(7, x.data_ptr(), y.data_ptr(), s)
        ctx.stream_wait(7, s)
    assert ctx.wait_all(10000) == nv.SUCCESS
    torch.cuda.synchronize()
    assert torch.equal(x, y)
    st = ctx.stats()
    assert (st["bytesReduced"], st["bytesCopied"]) == (4 * n * calls * reduced, 4 * n * calls * copied)
    assert st["deviceEvents"] >= 5 * calls
    ctx.trace_dump(str(tmp_path / "t.json"))
    names = [e["name"] for e in json.loads((tmp_path / "t.json").read_text())["traceEvents"] if e.get("args", {}).get("coll", 7) == 7]
    assert (names.count("sqe"), names.count("data"), names.count("done")) == (calls, 2 * calls, calls), names      # data: begin and end
    ctx.destroy()
    c.destroy()
