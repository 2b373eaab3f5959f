"""How long a wait of the scheduler lasts: without end while its collective is alone, until something else is submitted."""
import time

import numpy as np

from helpers import host_array, run_ranks
from test_host_runtime import _env


def test_a_wait_ends_when_something_else_is_submitted(host_backend):
    """Rank 0 waits in collective 0, for which its peer is not there, with more patience than the test lasts.  Collective 1 is
    submitted on both ranks and completes all the same; collective 0 does when the peer has come."""
    nv = host_backend
    comms = nv.Comm.init_loopback(2)
    first = [False]

    def body(r):
        ctx = nv.RankCtx(r)
        for i in range(2):
            ctx.prepare(i, comms[r], nv.ALLREDUCE, 5000, nv.FLOAT32, algo=nv.ALGO_TWOSHOT)
        ctx.finalize()
        p = [comms[r].alloc(20000) for _ in range(2)]
        for q in p:
            host_array(q, 5000, np.float32)[:] = r + 1
        if r == 0:
            ctx.run(0, p[0], p[0])
            time.sleep(0.3)                                # its blocks are in the wait by now
        ctx.run(1, p[1], p[1])
        assert ctx.wait(1, 30000) == nv.SUCCESS
        assert np.all(host_array(p[1], 5000, np.float32) == 3)
        if r == 0:
            first[0] = True
        else:
            while not first[0]:
                time.sleep(0.01)
            ctx.run(0, p[0], p[0])
        assert ctx.wait(0, 30000) == nv.SUCCESS
        assert np.all(host_array(p[0], 5000, np.float32) == 3)
        ctx.destroy()

    with _env(DFCCL_BASE_CTX_SWITCH_THRESHOLD=1 << 28, DFCCL_NUM_TRY_TASKQ_HEAD=5):
        run_ranks(2, body, timeout=120)
    for c in comms:
        c.destroy()
