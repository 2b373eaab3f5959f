"""A collective whose context a block still holds from its previous submission (csrc/src/device/daemon_impl.h:
consumeSubmissions) is submitted again.  Host backend; the scheduler is the same source as the device's."""
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
