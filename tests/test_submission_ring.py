"""The submission ring: entries carry a tag of their turn of the ring in every word (csrc/src/device/types.h), 127 turns
long; more submissions than that, and batches that fill several slots at once, must all arrive."""
import pytest

from helpers import run_ranks


def _case(nv, ranks, colls, rounds, count, alloc_view):
    comms = nv.Comm.init_loopback(ranks, 0)
    done = {}

    def body(r):
        c = comms[r]
        ctx = nv.RankCtx(r, 0)
        ctx.set_daemon_geometry(2, 0)
        for i in range(colls):
            ctx.prepare(i, c, nv.ALLREDUCE, count, nv.INT32)
        ctx.finalize()
        bufs = [(c.alloc(4 * count), c.alloc(4 * count)) for _ in range(colls)]
        views = [(alloc_view(s, count), alloc_view(d, count)) for s, d in bufs]
        for i, (s, _) in enumerate(views):
            s[:] = (r + 1) * (i + 1)
        for _ in range(rounds):
            for i in range(colls):
                ctx.run(i, *bufs[i])
            assert ctx.wait_all(60000) == nv.SUCCESS
        total = sum(q + 1 for q in range(ranks))
        assert all(int(d[0]) == int(d[count - 1]) == total * (i + 1) for i, (_, d) in enumerate(views))
        done[r] = ctx.stats()["cqesDelivered"]
        ctx.destroy()

    run_ranks(ranks, body, timeout=300)
    for c in comms:
        c.destroy()
    assert done == {r: colls * rounds for r in range(ranks)}


# a ring has at least 64 slots: 128 turns of it are 8192 entries.  (On the host backend every round is a hand-over between
# threads, a time slice each on a loaded machine: 8400 rounds of one entry took 30 s and more there, 640 of 13 a tenth.)
@pytest.mark.parametrize("ranks,colls,rounds", [(1, 13, 640), (2, 13, 700)])
def test_more_turns_than_tags_host(host_backend, ranks, colls, rounds):
    import numpy as np
    from helpers import host_array
    _case(host_backend, ranks, colls, rounds, 5, lambda p, n: host_array(p, n, np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("ranks,colls,rounds", [(1, 1, 8400), (2, 13, 700)])
def test_more_turns_than_tags_gpu(native, ranks, colls, rounds):
    import torch
    from dfccl_b200.utils import tensor_from_ptr
    native.set_backend("cuda")
    torch.cuda.set_device(0)

    class View:                                            # fills and reads on the default stream, finished before use
        def __init__(self, p, n):
            self.t = tensor_from_ptr(p, (n,), torch.int32, "cuda:0")

        def __setitem__(self, _, v):
            self.t.fill_(v)
            torch.cuda.current_stream().synchronize()

        def __getitem__(self, i):
            return self.t[i].item()

    _case(native, ranks, colls, rounds, 5, View)
