"""A collective whose context a block still holds from its previous submission (csrc/src/device/daemon_impl.h:
consumeSubmissions) is submitted again.  Most of it on the host backend: the scheduler is the same source as the device's."""
import threading
import time

import numpy as np
import pytest

from helpers import host_array, run_ranks
from test_host_runtime import _env

COUNT = 200000          # fp32 values: above the push limit, so the members read one another's heap


@pytest.mark.parametrize("algo", ["TWOSHOT", "ONESHOT"])
@pytest.mark.parametrize("then", ["xy", "py", "xq", "pp"])
def test_resubmission_that_needs_staging_areas(host_backend, algo, then):
    """Heap to heap three times, then, with the daemon resident all the while, from and / or to ordinary memory, or in place
    (one-shot: through a private copy of the input).  The blocks must hear of the staging areas made for it: the sums are
    right, and the front of the heap, where an area at offset 0 would lie, stays as it was."""
    nv = host_backend
    comms = nv.Comm.init_loopback(2)
    changed = {}

    def body(r):
        c = comms[r]
        ptr = {n: c.alloc(4 * COUNT) for n in "pq"}
        buf = {n: host_array(a, COUNT, np.float32) for n, a in ptr.items()}
        buf.update(x=np.zeros(COUNT, np.float32), y=np.zeros(COUNT, np.float32))
        ctx = nv.RankCtx(r)
        ctx.prepare(0, c, nv.ALLREDUCE, COUNT, nv.FLOAT32, algo=getattr(nv, "ALGO_" + algo))
        ctx.finalize()
        base = c.heap_info()[0]
        front = host_array(base, COUNT, np.float32)
        for it, (s, d) in enumerate(["pq"] * 3 + [then]):
            buf[s][:] = 10.0 * (r + 1) + it
            before = front.copy()
            ctx.run(0, buf[s].ctypes.data, buf[d].ctypes.data)
            assert ctx.wait(0, 30000) == nv.SUCCESS
            assert np.all(buf[d] == 30.0 + 2 * it), (it, buf[d][:3])
        diff = front.view(np.uint32) != before.view(np.uint32)
        for a in ptr.values():                   # (the user's own buffers may lie there)
            lo = max(0, (a - base) // 4)
            diff[lo:max(lo, (a - base) // 4 + COUNT)] = False
        changed[r] = int(diff.sum())
        ctx.destroy()
        for a in ptr.values():
            c.free(a)

    with _env(DFCCL_IDLE_QUIT_US=30000000, DFCCL_STALL_QUIT_US=30000000, DFCCL_MAX_LIFETIME_MS=0):
        run_ranks(2, body)
    for c in comms:
        c.destroy()
    assert all(n < 4096 for n in changed.values()), changed          # flag words


@pytest.mark.parametrize("count", [1000, COUNT])          # push and read schedules: the waits differ
def test_resubmission_that_stalls_lets_the_daemon_leave(host_backend, count):
    """One rank submits the id again and its peer comes 0.2 s late.  Stalled on the new epoch's flags (the previous epoch's are
    all there), the block must leave after the stall limit of 5 ms - again and again, since the work stays outstanding - and
    the peer's blocks, which share the launch, get in with the next one: not only after the lifetime limit, which is off."""
    nv = host_backend
    comms = nv.Comm.init_loopback(2)
    met = threading.Barrier(2)
    took, quits = {}, {}

    def body(r):
        c = comms[r]
        p, q = c.alloc(4 * count), c.alloc(4 * count)
        ctx = nv.RankCtx(r)
        ctx.prepare(0, c, nv.ALLREDUCE, count, nv.FLOAT32)
        ctx.finalize()
        host_array(p, count, np.float32)[:] = r + 1.0
        for _ in range(2):
            ctx.run(0, p, q)
            assert ctx.wait(0, 30000) == nv.SUCCESS
        met.wait()
        before = ctx.stats()["daemonVoluntaryQuits"]
        if r == 1:
            time.sleep(0.2)
        t = time.perf_counter()
        ctx.run(0, p, q)
        assert ctx.wait(0, 10000) == nv.SUCCESS
        took[r] = time.perf_counter() - t
        quits[r] = ctx.stats()["daemonVoluntaryQuits"] - before
        assert np.all(host_array(q, count, np.float32) == 3.0)
        ctx.destroy()

    with _env(DFCCL_DAEMON_BLOCKS=1, DFCCL_IDLE_QUIT_US=1000, DFCCL_STALL_QUIT_US=5000, DFCCL_MAX_LIFETIME_MS=0):
        run_ranks(2, body)
    for c in comms:
        c.destroy()
    assert quits[0] >= 2 and took[1] < 2.0, (quits, took)


@pytest.mark.gpu
@pytest.mark.parametrize("then", ["xy", "pp"])
def test_resubmission_that_needs_staging_areas_gpu(native, then):
    """One-shot; the daemon stays for 0.2 s, far longer than the four submissions take."""
    import torch
    from dfccl_b200.utils import tensor_from_ptr
    native.set_backend("cuda")
    torch.cuda.set_device(0)
    comms = native.Comm.init_loopback(2, 0)
    buf = [{n: tensor_from_ptr(comms[r].alloc(4 * COUNT), (COUNT,), torch.float32, "cuda:0") for n in "pq"} |
           {n: torch.zeros(COUNT, device="cuda") for n in "xy"} for r in range(2)]
    torch.cuda.synchronize()

    def body(r):
        torch.cuda.set_device(0)
        ctx = native.RankCtx(r, 0)
        ctx.set_daemon_geometry(2, 0)
        ctx.prepare(0, comms[r], native.ALLREDUCE, COUNT, native.FLOAT32, algo=native.ALGO_ONESHOT)
        ctx.finalize()
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            for it, (s, d) in enumerate(["pq"] * 3 + [then]):
                buf[r][s].fill_(10.0 * (r + 1) + it)
                st.synchronize()
                ctx.run(0, buf[r][s].data_ptr(), buf[r][d].data_ptr())
                assert ctx.wait(0, 30000) == native.SUCCESS
                assert bool((buf[r][d] == 30.0 + 2 * it).all()), it
        ctx.destroy()

    with _env(DFCCL_IDLE_QUIT_US=200000, DFCCL_STALL_QUIT_US=200000):
        run_ranks(2, body)
    for c in comms:
        c.destroy()


@pytest.mark.gpu
def test_resubmission_with_a_late_peer_gpu(native):
    """With the default limits (a stalled block leaves after 5 ms, any daemon after 2 s)."""
    import torch
    from dfccl_b200.utils import tensor_from_ptr
    native.set_backend("cuda")
    torch.cuda.set_device(0)
    comms = native.Comm.init_loopback(2, 0)
    met = threading.Barrier(2)
    took = {}

    def body(r):
        torch.cuda.set_device(0)
        c = comms[r]
        p, q = c.alloc(4 * COUNT), c.alloc(4 * COUNT)
        x, y = (tensor_from_ptr(a, (COUNT,), torch.float32, "cuda:0") for a in (p, q))
        ctx = native.RankCtx(r, 0)
        ctx.set_daemon_geometry(2, 0)
        ctx.prepare(0, c, native.ALLREDUCE, COUNT, native.FLOAT32)
        ctx.finalize()
        x.fill_(r + 1.0)
        torch.cuda.current_stream().synchronize()
        for _ in range(2):
            ctx.run(0, p, q)
            assert ctx.wait(0, 30000) == native.SUCCESS
        met.wait()
        if r == 1:
            time.sleep(0.1)
        t = time.perf_counter()
        ctx.run(0, p, q)
        assert ctx.wait(0, 30000) == native.SUCCESS
        took[r] = time.perf_counter() - t
        assert bool((y == 3.0).all())
        ctx.destroy()

    run_ranks(2, body)
    for c in comms:
        c.destroy()
    assert took[1] < 0.5, took
