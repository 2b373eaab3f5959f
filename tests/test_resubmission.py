"""A collective whose context a block still holds from its previous submission (csrc/src/device/daemon_impl.h:
consumeSubmissions) is submitted again.  Host backend; the scheduler is the same source as the device's."""
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
