"""Daemon blocks of other than the default number of threads; their last warp is the service warp."""
import pytest
import torch

from helpers import run_ranks
from test_host_runtime import _env

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 32, 33, 100, 480, 511, 512])
def test_daemon_blocks_of_any_number_of_threads(native, threads):
    from dfccl_b200.utils import tensor_from_ptr
    native.set_backend("cuda")
    torch.cuda.set_device(0)
    n = 100003
    with _env(DFCCL_DAEMON_THREADS=threads):
        comms = native.Comm.init_loopback(2, 0)

        def body(r):
            c = comms[r]
            ctx = native.RankCtx(r, 0)
            ctx.set_daemon_geometry(2, 0)
            ctx.prepare(0, c, native.ALLREDUCE, n, native.FLOAT32)
            ctx.prepare(1, c, native.ALLREDUCE, 509, native.FLOAT32)
            ctx.finalize()
            bufs = [(c.alloc(4 * m), c.alloc(4 * m), m) for m in (n, 509)]
            views = [(tensor_from_ptr(p, (m,), torch.float32, "cuda:0"), tensor_from_ptr(q, (m,), torch.float32, "cuda:0")) for p, q, m in bufs]
            for it in range(3):
                for x, _ in views:
                    x.fill_(float(r + 1 + it))
                torch.cuda.current_stream().synchronize()
                for i, (p, q, _) in enumerate(bufs):
                    ctx.run(i, p, q)
                assert ctx.wait_all(60000) == native.SUCCESS
                for _, y in views:
                    assert bool((y == 3.0 + 2 * it).all())
            ctx.destroy()

        run_ranks(2, body)
        for c in comms:
            c.destroy()
