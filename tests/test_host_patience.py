"""How long a wait of the scheduler lasts: while its collective is alone, until something else is submitted."""
import time

import numpy as np
import pytest

from helpers import host_array, run_ranks
from test_host_runtime import _env


@pytest.mark.parametrize("on_stream", [False, True])
def test_a_wait_ends_when_something_else_is_submitted(host_backend, on_stream):
    """Rank 0's only block waits in collective 0, for which its peer is not there, for 4e9 polls (13 s, at 3.3 ns).  Collective 1 is
    submitted on both ranks, directly or to be released by a stream (an eighth of the polls), and is complete long before; collective
    0 when the peer has come."""
    nv = host_backend
    comms = nv.Comm.init_loopback(2)
    took = {}

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
            time.sleep(0.3)                                # its block is in the wait by now
        t0 = time.time()
        if on_stream:
            ctx.run_on_stream(1, p[1], p[1], 0)
        else:
            ctx.run(1, p[1], p[1])
        assert ctx.wait(1, 60000) == nv.SUCCESS
        took[r] = time.time() - t0
        assert np.all(host_array(p[1], 5000, np.float32) == 3)
        if r == 1:
            while 0 not in took:
                time.sleep(0.01)
            ctx.run(0, p[0], p[0])
        assert ctx.wait(0, 60000) == nv.SUCCESS
        assert np.all(host_array(p[0], 5000, np.float32) == 3)
        ctx.destroy()

    # beside another collective a wait is a sixteenth of the threshold: 4e6 polls
    with _env(DFCCL_BASE_CTX_SWITCH_THRESHOLD=1 << 26, DFCCL_NUM_TRY_TASKQ_HEAD=60, DFCCL_DAEMON_BLOCKS=1, DFCCL_IDLE_QUIT_US=10 ** 8,
              DFCCL_STALL_QUIT_US=10 ** 8, DFCCL_MAX_LIFETIME_MS=10 ** 6):
        run_ranks(2, body, timeout=120)
    assert took[0] < 6, took
    for c in comms:
        c.destroy()
