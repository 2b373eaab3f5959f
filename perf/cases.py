"""What the framework is measured on: the work a program hands to it on one GPU, through its public entry points.

Eight kinds of work, over their ranges:

  submit   one registered all-reduce per pass through the daemon, several ranks on one device (the loopback group of the
           tests): register once, then submit from the host on every rank and wait
  shards   the exchange of a sharded optimizer: reduce-scatter of fp32 gradients, then all-gather of bf16 parameters
  disorder a batch of collectives of mixed kinds and sizes that every rank submits in an order of its own
  stream   several registered all-reduces of a one-rank job in flight on one stream: stream-ordered submit and wait
  nccl     a stream-ordered collective on ordinary tensors (not in the symmetric heap) of a one-rank job
  gemm     products of a linear layer on the tensor-core kernel: forward, data gradient and weight gradient
  ddp      gradients of a model through ``DaemonDDP``: bucket all-reduce, then the fused optimizer step
  blocks   a whole training step of the middle pipeline stage of GPT-2: forward, backward, gradient buckets, AdamW

``prepare`` keeps what a program keeps: communicators and rank contexts (one set per process, registered once), buffers
in the symmetric heap, modules and their optimizer state.
"""
from __future__ import annotations

import os
import random
import threading
import weakref

import torch
import torch.nn as nn

from dfccl_b200 import native as nv
from dfccl_b200.models.gpt2 import GPT2Config, GPT2Stage
from dfccl_b200.models.resnet import resnet50, to_bf16_channels_last
from dfccl_b200.ops import collectives, gemm
from dfccl_b200.ops.fused_linear import TpGroup
from dfccl_b200.parallel import DaemonDDP
from dfccl_b200.parallel.groups import Dist
from dfccl_b200.utils.tensors import nccl_dtype, tensor_from_ptr

# waits of the daemon end with an error status instead of lasting for ever, as in the benchmarks
os.environ.setdefault("DFCCL_WAIT_TIMEOUT_MS", "60000")

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "int32": torch.int32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4, "int32": 4}
OPS = {"sum": nv.SUM, "max": nv.MAX, "avg": nv.AVG}
KINDS = {"allreduce": nv.ALLREDUCE, "allgather": nv.ALLGATHER, "reducescatter": nv.REDUCESCATTER, "broadcast": nv.BROADCAST}
WAIT_MS = 60000


def listed():
    return [
        # a scalar-sized reduction among four ranks (a loss, a norm, a flag): latency only, an odd length
        {"name": "submit_small", "family": "submit", "ranks": 4, "count": 509, "dtype": "bf16", "out": "bf16", "op": "sum", "scale": 1.0},
        # one 25 MiB gradient bucket among four ranks: bf16 in, fp32 average out (scale and cast inside the collective)
        {"name": "submit_bucket", "family": "submit", "ranks": 4, "count": 13107200, "dtype": "bf16", "out": "fp32", "op": "sum", "scale": 0.25},
        # sharded optimizer, ragged shard length: gradients reduce-scattered in fp32, parameters gathered in bf16
        {"name": "shards_ragged", "family": "shards", "ranks": 4, "count": 250003},
        # the disordered-issue workload: 24 collectives of mixed kinds, 1 K to 1 M elements, every rank its own order
        {"name": "disorder_24", "family": "disorder", "ranks": 4, "colls": 24, "low": 1024, "high": 1048576, "plan": 3},
        # one-rank job, stream-ordered: eight messages of 64 KB in flight, released and awaited by the stream
        {"name": "stream_64k", "family": "stream", "ids": 8, "count": 32768, "dtype": "bf16", "out": "bf16"},
        # ordinary tensors of a one-rank job, ragged length, averaged in fp32
        {"name": "nccl_tensors", "family": "nccl", "kind": "allreduce", "count": 8388611, "dtype": "fp32", "op": "avg"},
        # smallest product of the tensor-core kernel that is used in earnest: one row tile, short contraction
        {"name": "gemm_small", "family": "gemm", "m": 128, "n": 512, "k": 512},
        # odd multiples of the tile: 15 row tiles, 5 column tiles, 12 contraction steps
        {"name": "gemm_ragged", "family": "gemm", "m": 1920, "n": 1280, "k": 768},
        # the up projection of GPT-2 medium (1024 -> 4096) on 8 sequences of 1024 tokens
        {"name": "gemm_layer", "family": "gemm", "m": 8192, "n": 4096, "k": 1024},
        # the size at which the GEMM benchmark quotes its throughput
        {"name": "gemm_8192", "family": "gemm", "m": 8192, "n": 8192, "k": 8192},
        # ResNet-50 data parallel: 25 MB buckets, all-reduce with fused scale and cast, fused SGD on fp32 master weights
        {"name": "ddp_resnet50", "family": "ddp", "params": 0, "bucket_mb": 25.0, "optimizer": "sgd"},
        # GPT-2 medium cut into eight pipeline stages: three blocks on 8 sequences of 1024 tokens, AdamW
        {"name": "blocks_medium", "family": "blocks", "layers": 3, "d": 1024, "heads": 16, "seq": 1024, "micro": 8},
    ]


def _log(rng, low, high):
    """Log-uniform whole number of [low, high]."""
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    family = rng.choice(["submit", "submit", "shards", "disorder", "stream", "nccl", "gemm", "gemm", "gemm", "ddp", "blocks"])
    if family == "submit":
        dtype, out, op, scale = rng.choice([("bf16", "bf16", "sum", 1.0), ("bf16", "fp32", "sum", 0.25), ("fp32", "fp32", "avg", 1.0),
                                            ("fp16", "fp16", "sum", 1.0), ("fp32", "fp32", "max", 1.0), ("int32", "int32", "sum", 1.0)])
        ranks = rng.choice([2, 4, 8])
        return {"family": family, "ranks": ranks, "count": _log(rng, 256, 16 << 20), "dtype": dtype, "out": out, "op": op, "scale": scale}
    if family == "shards":
        return {"family": family, "ranks": rng.choice([2, 4]), "count": _log(rng, 4096, 2 << 20)}
    if family == "disorder":
        return {"family": family, "ranks": rng.choice([2, 4]), "colls": rng.randint(8, 32), "low": 1024, "high": _log(rng, 1 << 15, 2 << 20),
                "plan": rng.randint(1, 1 << 20)}
    if family == "stream":
        dtype, out = rng.choice([("bf16", "bf16"), ("bf16", "fp32"), ("fp32", "fp32")])
        return {"family": family, "ids": rng.randint(1, 8), "count": _log(rng, 512, 8 << 20), "dtype": dtype, "out": out}
    if family == "nccl":
        return {"family": family, "kind": rng.choice(["allreduce", "allgather", "reducescatter"]), "count": _log(rng, 1024, 32 << 20),
                "dtype": rng.choice(["fp32", "bf16"]), "op": rng.choice(["sum", "avg"])}
    if family == "gemm":
        # half of the contractions are multiples of 256, so that the gradients' products tile too
        k = rng.choice([64 * _log(rng, 4, 128), 256 * _log(rng, 1, 32)])
        return {"family": family, "m": 128 * _log(rng, 1, 64), "n": 256 * _log(rng, 1, 32), "k": k}
    if family == "ddp":
        return {"family": family, "params": _log(rng, 1 << 20, 32 << 20), "bucket_mb": 25.0, "optimizer": rng.choice(["sgd", "adamw"])}
    d = rng.choice([256, 512, 1024])
    return {"family": family, "layers": rng.randint(1, 3), "d": d, "heads": d // 64, "seq": rng.choice([128, 256, 512, 1024]), "micro": rng.randint(2, 8)}


# ---------------------------------------------------------------------------------------------- one group per process
class Group:
    """Loopback communicators of ``ranks`` ranks on one device, and a rank context each with ``colls`` registered."""

    def __init__(self, ranks, colls):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.comms = nv.Comm.init_loopback(ranks, self.device.index)
        self.ctxs = []
        if not colls:
            return
        for r, comm in enumerate(self.comms):
            ctx = nv.RankCtx(r, self.device.index)
            ctx.set_daemon_geometry(min(32, 128 // ranks), 0)
            for i, (kind, count, dtype, out, op, scale, root) in enumerate(colls):
                ctx.prepare(i, comm, kind, count, nccl_dtype(DTYPES[dtype]), out_dtype=nccl_dtype(DTYPES[out]), op=op, root=root, scale=scale)
            self.ctxs.append(ctx)
        failed = []

        def finalize(ctx):
            try:
                torch.cuda.set_device(self.device)
                ctx.finalize()
            except Exception as e:                       # raised again below, in the caller's thread
                failed.append(e)

        threads = [threading.Thread(target=finalize, args=(c,)) for c in self.ctxs]      # the ranks meet here
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        if failed:
            raise failed[0]

    def buffer(self, rank, count, dtype):
        """(address, tensor) of ``count`` elements in the symmetric heap of ``rank``."""
        p = self.comms[rank].alloc(max(16, count * BYTES[dtype]))
        return p, tensor_from_ptr(p, (count,), DTYPES[dtype], self.device)

    def close(self):
        torch.cuda.synchronize()
        for c in self.ctxs:
            c.destroy()
        for c in self.comms:
            c.destroy()


_group = {"key": None, "group": None}
_states = weakref.WeakSet()


def _group_of(ranks, colls):
    """The process's group: made on first use, made anew when another set of collectives is asked for."""
    key = (ranks, tuple(colls))
    if _group["key"] != key:
        for s in list(_states):
            s.release()
        if _group["group"] is not None:
            _group["group"].close()
        _group["key"], _group["group"] = None, None
        _group["group"], _group["key"] = Group(ranks, colls), key
    return _group["group"]


class State:
    """What a pass runs on; ``release`` gives back what the Python objects do not own."""

    def __init__(self, **kw):
        self.__dict__.update(kw)
        self.held = kw.get("held", [])                   # (communicator, heap address)
        self.closers = kw.get("closers", [])
        _states.add(self)

    def release(self):
        held, self.held = self.held, []
        closers, self.closers = self.closers, []
        if held:
            torch.cuda.synchronize()
        for comm, p in held:
            comm.free(p)
        for f in closers:
            f()

    def __del__(self):
        try:
            self.release()
        except Exception:
            pass


def _values(gen, count, dtype, device, scale=1.0):
    if dtype == "int32":
        return torch.randint(-1000, 1001, (count,), generator=gen, device=device, dtype=torch.int32)
    return torch.randn(count, generator=gen, device=device).mul_(scale).to(DTYPES[dtype])


# ---------------------------------------------------------------------------------------------- prepare
def _disorder_plan(case):
    """[(kind, count, root)]: the same on every rank."""
    rng = random.Random(case["plan"])
    plan = []
    for i in range(case["colls"]):
        kind = rng.choice(["allreduce", "allgather", "reducescatter", "broadcast"])
        count = _log(rng, case["low"], case["high"])
        if kind in ("allgather", "reducescatter"):
            count = max(16, count // case["ranks"])
        plan.append((kind, count, i % case["ranks"]))
    return plan


def _lengths(kind, count, ranks):
    return count * (ranks if kind == "reducescatter" else 1), count * (ranks if kind == "allgather" else 1)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    nv.set_backend("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    return globals()["_prepare_" + case["family"]](case, seed, gen, dev)


def _prepare_submit(case, seed, gen, dev):
    group = _group_of(case["ranks"], [(nv.ALLREDUCE, case["count"], case["dtype"], case["out"], OPS[case["op"]], case["scale"], 0)])
    held, calls, outs = [], [], []
    for r, comm in enumerate(group.comms):
        sp, x = group.buffer(r, case["count"], case["dtype"])
        rp, y = group.buffer(r, case["count"], case["out"])
        x.copy_(_values(gen, case["count"], case["dtype"], dev))
        y.zero_()
        held += [(comm, sp), (comm, rp)]
        calls.append((group.ctxs[r], sp, rp))
        outs.append(y)
    return State(run=_run_submit, calls=calls, outs=outs, held=held)


def _prepare_shards(case, seed, gen, dev):
    n, ranks = case["count"], case["ranks"]
    group = _group_of(ranks, [(nv.REDUCESCATTER, n, "fp32", "fp32", nv.SUM, 1.0, 0), (nv.ALLGATHER, n, "bf16", "bf16", nv.SUM, 1.0, 0)])
    held, calls, outs = [], [], []
    for r, comm in enumerate(group.comms):
        gp, g = group.buffer(r, n * ranks, "fp32")
        sp, s = group.buffer(r, n, "fp32")
        pp, p = group.buffer(r, n, "bf16")
        fp, f = group.buffer(r, n * ranks, "bf16")
        g.copy_(_values(gen, n * ranks, "fp32", dev, 1e-2))
        p.copy_(_values(gen, n, "bf16", dev, 2e-2))
        s.zero_()
        f.zero_()
        held += [(comm, q) for q in (gp, sp, pp, fp)]
        calls.append((group.ctxs[r], gp, sp, pp, fp))
        outs += [s, f]
    return State(run=_run_shards, calls=calls, outs=outs, held=held)


def _prepare_disorder(case, seed, gen, dev):
    ranks, plan = case["ranks"], _disorder_plan(case)
    group = _group_of(ranks, [(KINDS[k], n, "bf16", "bf16", nv.SUM, 1.0, root) for k, n, root in plan])
    held, calls, outs = [], [], []
    for r, comm in enumerate(group.comms):
        # one allocation per direction: the collectives' buffers follow one another in it, 512 bytes apart
        total = [0, 0]
        offs = []
        for k, n, _ in plan:
            sn, rn = _lengths(k, n, ranks)
            offs.append((total[0], total[1]))
            total[0] += (sn + 255) // 256 * 256
            total[1] += (rn + 255) // 256 * 256
        sp, x = group.buffer(r, total[0], "bf16")
        rp, y = group.buffer(r, total[1], "bf16")
        x.copy_(_values(gen, total[0], "bf16", dev))
        y.zero_()
        held += [(comm, sp), (comm, rp)]
        order = list(range(len(plan)))
        random.Random(1000 * seed + r).shuffle(order)
        calls.append((group.ctxs[r], [(i, sp + 2 * offs[i][0], rp + 2 * offs[i][1]) for i in order]))
        outs.append(y)
    return State(run=_run_disorder, calls=calls, outs=outs, held=held)


def _prepare_stream(case, seed, gen, dev):
    n = case["count"]
    group = _group_of(1, [(nv.ALLREDUCE, n, case["dtype"], case["out"], nv.SUM, 0.5, 0)] * case["ids"])
    held, calls, outs = [], [], []
    for i in range(case["ids"]):
        sp, x = group.buffer(0, n, case["dtype"])
        rp, y = group.buffer(0, n, case["out"])
        x.copy_(_values(gen, n, case["dtype"], dev))
        y.zero_()
        held += [(group.comms[0], sp), (group.comms[0], rp)]
        calls.append((i, sp, rp))
        outs.append(y)
    return State(run=_run_stream, ctx=group.ctxs[0], calls=calls, outs=outs, held=held)


def _prepare_nccl(case, seed, gen, dev):
    group = _group_of(1, [])
    x = _values(gen, case["count"], case["dtype"], dev)
    return State(run=_run_nccl, comm=group.comms[0], kind=case["kind"], op=case["op"], x=x, out=torch.zeros_like(x))


def _prepare_gemm(case, seed, gen, dev):
    m, n, k = case["m"], case["n"], case["k"]
    x = torch.randn(m, k, generator=gen, device=dev).to(torch.bfloat16)                      # activations of the layer
    w = (torch.randn(n, k, generator=gen, device=dev) * k ** -0.5).to(torch.bfloat16)        # its weight, as nn.Linear stores it
    gy = torch.randn(m, n, generator=gen, device=dev).to(torch.bfloat16)                     # gradient of its output
    empty = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device=dev)                     # noqa: E731
    # the products whose sizes tile: the forward pass always does, the gradients where k and m are multiples of the tile
    dgrad, wgrad = gemm.gemm_supported(m, k, n), gemm.gemm_supported(n, k, m)
    return State(run=_run_gemm, x=x, w=w, gy=gy, y=empty(m, n), gx=empty(m, k) if dgrad else None, gw=empty(n, k) if wgrad else None)


class _Stack(nn.Module):
    """``total`` parameters in square-ish matrices with a bias each, as a stack of linear layers holds them."""

    def __init__(self, total, device):
        super().__init__()
        ps, left = [], total
        while left > 0:
            n = min(left, 1 << 20)
            side = max(1, int(n ** 0.5))
            ps.append(nn.Parameter(torch.zeros(side, max(1, n // side), dtype=torch.bfloat16, device=device)))
            ps.append(nn.Parameter(torch.zeros(side, dtype=torch.bfloat16, device=device)))
            left -= ps[-2].numel() + side
        self.ps = nn.ParameterList(ps)


def _dist(dev):
    (comm,) = nv.Comm.init_loopback(1, dev.index)
    return Dist(0, 1, dev.index, dev, comm, False)


def _close_ddp(ddp, d):
    ddp.close()
    d.comm.destroy()


def _prepare_ddp(case, seed, gen, dev):
    if case["params"]:
        net = _Stack(case["params"], dev)
    else:
        with dev:
            net = to_bf16_channels_last(resnet50(1000))
    with torch.no_grad():
        for p in net.parameters():
            p.copy_(torch.randn(p.shape, generator=gen, device=dev) * 0.02)
    d = _dist(dev)
    ddp = DaemonDDP(net, d, bucket_mb=case["bucket_mb"], lr=0.1 if case["optimizer"] == "sgd" else 1e-3, optimizer=case["optimizer"], seed=17)
    grads = [torch.randn(b.numel, generator=gen, device=dev).mul_(1e-2).to(b.dtype) for b in ddp.buckets]
    return State(run=_run_ddp, net=net, ddp=ddp, grads=grads, closers=[lambda: _close_ddp(ddp, d)])


def _prepare_blocks(case, seed, gen, dev):
    d = _dist(dev)
    tp = TpGroup(d.comm, None, dev, ctx=nv.RankCtx(0, dev.index))
    cfg = GPT2Config(n_layer=3 * case["layers"], d_model=case["d"], n_head=case["heads"], seq_len=case["seq"])
    stage = GPT2Stage(cfg, tp, 1, 3, case["micro"], seed=seed)
    with torch.no_grad():                                # norms and biases off their initial ones and zeros, as in training
        for p in stage.parameters():
            if p.dim() == 1:
                p.add_((torch.randn(p.shape, generator=gen, device=dev) * 0.02).to(p.dtype))
    # the step size of the first AdamW step is lr for every weight: small against weights of 0.02
    ddp = DaemonDDP(stage, d, lr=1e-5, weight_decay=0.01, optimizer="adamw", seed=17, ctx=tp.ctx, coll_id_base=tp.next_id)
    shape = (stage.rows, cfg.d_model)
    x = torch.randn(shape, generator=gen, device=dev).to(torch.bfloat16).requires_grad_(True)
    gy = (torch.randn(shape, generator=gen, device=dev) / stage.tokens).to(torch.bfloat16)
    return State(run=_run_blocks, stage=stage, ddp=ddp, x=x, gy=gy, done=None, closers=[lambda: _close_ddp(ddp, d)])


# ---------------------------------------------------------------------------------------------- run
def run(state):
    return state.run(state)


def _wait(ctx, i):
    nv.check(ctx.wait(i, WAIT_MS), "wait")


def _run_submit(s):
    for ctx, sp, rp in s.calls:
        ctx.run(0, sp, rp)
    for ctx, _, _ in s.calls:
        _wait(ctx, 0)
    return s.outs


def _run_shards(s):
    for ctx, gp, sp, _, _ in s.calls:
        ctx.run(0, gp, sp)
    for ctx, _, _, pp, fp in s.calls:
        _wait(ctx, 0)                                    # (where a real step updates its shard of the parameters)
        ctx.run(1, pp, fp)
    for ctx, *_ in s.calls:
        _wait(ctx, 1)
    return s.outs


def _run_disorder(s):
    for ctx, subs in s.calls:
        for i, sp, rp in subs:
            ctx.run(i, sp, rp)
    for ctx, _ in s.calls:
        nv.check(ctx.wait_all(WAIT_MS), "wait_all")
    return s.outs


def _run_stream(s):
    st = torch.cuda.current_stream().cuda_stream
    for i, sp, rp in s.calls:
        s.ctx.run_on_stream(i, sp, rp, st)
    for i, _, _ in s.calls:
        s.ctx.stream_wait(i, st)
    return s.outs


def _run_nccl(s):
    if s.kind == "allreduce":
        return collectives.all_reduce(s.comm, s.x, s.out, op=s.op)
    if s.kind == "allgather":
        return collectives.all_gather(s.comm, s.x, s.out)
    return collectives.reduce_scatter(s.comm, s.x, s.out, op=s.op)


def _run_gemm(s):
    outs = [gemm.matmul_nt(s.x, s.w, s.y)]                                                    # y = x W^T
    if s.gx is not None:
        outs.append(gemm.matmul(s.gy, s.w, s.gx, b_transposed=True))                          # gx = gy W
    if s.gw is not None:
        outs.append(gemm.matmul(s.gy, s.x, s.gw, a_transposed=True, b_transposed=True))       # gW = gy^T x
    return outs


def _run_ddp(s):
    for b, g in zip(s.ddp.buckets, s.grads):             # stands for the backward pass, which fills the buckets
        b.grad.copy_(g)
    s.ddp.finish_backward()
    s.ddp.step()
    return {"master": [b.master for b in s.ddp.buckets], "momentum": [b.momentum for b in s.ddp.buckets],
            "param": [b.flat_param for b in s.ddp.buckets]}


def _run_blocks(s):
    if s.done is not None:                               # the trainer keeps the host within one step of the GPU
        s.done.synchronize()
    s.x.grad = None
    y = s.stage(s.x)
    y.backward(s.gy)
    s.ddp.finish_backward()
    s.ddp.step()
    s.done = torch.cuda.Event()
    s.done.record()
    return {"y": y.detach(), "gx": s.x.grad, "master": [b.master for b in s.ddp.buckets], "momentum": [b.momentum for b in s.ddp.buckets],
            "param": [b.flat_param for b in s.ddp.buckets]}


# ---------------------------------------------------------------------------------------------- work and tolerance
RESNET50_PARAMS = 25557032


def work(case):
    f = case["family"]
    if f == "submit":
        n = case["count"] * case["ranks"]
        return {"bytes": n * (BYTES[case["dtype"]] + BYTES[case["out"]]), "flops": n}
    if f == "shards":
        n, r = case["count"], case["ranks"]
        return {"bytes": r * (n * r * 4 + n * 4 + n * 2 + n * r * 2), "flops": n * r * (r - 1)}
    if f == "disorder":
        r, total = case["ranks"], 0
        for kind, n, _ in _disorder_plan(case):
            sn, rn = _lengths(kind, n, r)
            total += 2 * ((sn if kind == "broadcast" else r * sn) + r * rn)
        return {"bytes": total, "flops": 0}
    if f == "stream":
        return {"bytes": case["ids"] * case["count"] * (BYTES[case["dtype"]] + BYTES[case["out"]]), "flops": 0}
    if f == "nccl":
        return {"bytes": 2 * case["count"] * BYTES[case["dtype"]], "flops": 0}
    if f == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        each = 2 * (m * k + n * k + m * n)
        products = 1 + int(m % 128 == 0 and k % 256 == 0 and n % 64 == 0) + int(n % 128 == 0 and k % 256 == 0 and m % 64 == 0)
        return {"bytes": products * each, "flops": products * 2 * m * n * k}
    if f == "ddp":
        n = case["params"] or RESNET50_PARAMS
        # gradient in bf16; fp32 weights and moments read and written; bf16 parameters written
        return {"bytes": n * (2 + (16 if case["optimizer"] == "sgd" else 24) + 2), "flops": 4 * n}
    d, tokens = case["d"], case["seq"] * case["micro"]
    n = case["layers"] * 12 * d * d
    attention = case["layers"] * 3.5 * 4 * tokens * case["seq"] * d / 2
    return {"bytes": n * 28 + 4 * tokens * d * 2, "flops": 6 * n * tokens + attention}


def tolerance(case):
    """Four times what another correct order of the same sums was seen to change, with room for longer sums."""
    f = case["family"]
    if f == "shards":                                    # up to four fp32 values (4e-8 from their sum in 64 bits); copies
        return {"rel": 1e-6}
    if f in ("submit", "stream", "nccl", "disorder"):
        kind = case.get("out", case.get("dtype", "bf16"))
        if kind == "int32" or case.get("op") == "max":
            return "exact"
        # one rounding of a sum in fp32: another order moves a few results by one unit in the last place
        return {"bf16": {"rel": 1e-3}, "fp16": {"rel": 2e-4}, "fp32": {"rel": 1e-6}}[kind]
    if f == "gemm":                                      # fp32 sums rounded to bf16 once (4e-5 at k = 512, grows with k)
        return {"rel": 1e-3}
    if f == "ddp":                                       # fp32 arithmetic; bf16 parameters may differ by one unit in the last place
        return {"rel": 1e-5, "max": 1e-2}
    # bf16 activations through whole layers: 2.6e-3 (output), 4.9e-3 (gradients) with the biases added before the rounding
    return {"rel": 1e-2}
