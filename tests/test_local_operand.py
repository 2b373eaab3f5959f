"""What a one-rank fused operator (ops/fused_linear.py) hands to its GEMM, which takes bare pointers: operands of the
declared size and type whatever it was called with.  The library is a recorder here."""
import ctypes as C
from types import SimpleNamespace

import pytest
import torch

from dfccl_b200.ops import block, fused_linear

M, K, N = 128, 64, 256


class Recorder:
    """Stands for the library: notes the product's operands as the kernel would read them."""

    def __init__(self):
        self.calls = []

    def dfcclGemmBf16Epilogue(self, x, w, out, m, n, k, *rest):
        assert (x | w | out) % 16 == 0
        read = lambda p, rows, cols: torch.frombuffer((C.c_char * (2 * rows * cols)).from_address(p), dtype=torch.bfloat16).view(rows, cols).clone()   # noqa: E731
        self.calls.append((read(x, m, k), read(w, n, k), rest))
        return 0


@pytest.fixture()
def op(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(fused_linear.nv, "lib", lambda: rec)
    monkeypatch.setattr(fused_linear, "raw_stream", lambda _d: 0)
    o = fused_linear.AllGatherGemm.__new__(fused_linear.AllGatherGemm)
    o.tp, o.m, o.rows, o.k, o.n_out, o.coll_id = SimpleNamespace(n=1, device=torch.device("cpu")), M, M, K, N, None
    o.rec = rec
    return o


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("form", ["rows", "strided", "flat", "row", "vector", "off"])
def test_operand_is_cast_and_spread_like_a_copy(op, dtype, form):
    x = torch.randn(M, K).to(dtype)
    want = x
    if form == "strided":
        x = x.t().contiguous().t()
    elif form == "off":                                    # one element behind the 16-byte grid
        x = torch.cat([x.reshape(-1)[:1], x.reshape(-1)])[1:].view(M, K)
    elif form == "flat":
        x = x.view(2, M // 2, K)
    elif form in ("row", "vector"):
        x = x[:1] if form == "row" else x[0]
        want = x.expand(M, K)
    w = torch.randn(N, K).to(dtype)
    op.local(x, w)
    (got_x, got_w, _), = op.rec.calls
    assert torch.equal(got_x, want.to(torch.bfloat16)) and torch.equal(got_w, w.to(torch.bfloat16))


@pytest.mark.parametrize("xs,ws", [((M - 1, K), (N, K)), ((M, K // 2), (N, K)), ((M // 2, 2 * K), (N, K)), ((M, K), (N - 1, K)), ((M, K), (K, N))])
def test_operands_of_another_size_do_not_reach_the_kernel(op, xs, ws):
    with pytest.raises((ValueError, RuntimeError)):
        op.local(torch.zeros(xs, dtype=torch.bfloat16), torch.zeros(ws, dtype=torch.bfloat16))
    assert not op.rec.calls


BF = torch.bfloat16


@pytest.mark.parametrize("t,ok", [(torch.zeros(M, N, dtype=BF), True), (torch.zeros(N, M, dtype=BF).t(), True), (torch.zeros(M, N), False),
                                  (torch.zeros(1, N, dtype=BF), False), (torch.zeros(N, dtype=BF), False), (torch.zeros(M, 1, dtype=BF), False),
                                  (torch.zeros(M + 1, N, dtype=BF), False), (torch.zeros(M * N + 1, dtype=BF)[1:].view(M, N), False), (None, False)])
def test_which_residuals_ride_in_an_epilogue(t, ok):
    assert block.epilogue_operand(t, (M, N), torch.device("cpu")) == ok


@pytest.mark.parametrize("kw", [dict(bias=torch.zeros(1, dtype=BF)), dict(bias=torch.zeros(N, dtype=BF), aux=torch.zeros(1, N, dtype=BF)),
                                dict(bias=torch.zeros(N, dtype=BF), aux=torch.zeros(M - 1, N, dtype=BF)),
                                dict(bias=torch.zeros(N, dtype=BF), pre=torch.zeros(M, N - 8, dtype=BF))])
def test_epilogue_operands_of_another_shape_do_not_reach_the_kernel(op, kw):
    with pytest.raises(ValueError):
        op.local(torch.zeros(M, K, dtype=BF), torch.zeros(N, K, dtype=BF), epi=block.Epilogue(block.BIAS_RES, **kw))
    with pytest.raises(ValueError):
        block.apply_epilogue_(torch.zeros(M, N, dtype=BF), block.Epilogue(block.BIAS_RES, **kw))
    assert not op.rec.calls


def test_launches_on_a_device_that_is_not_current(monkeypatch):
    import contextlib
    from dfccl_b200.utils.tensors import on_device
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    assert isinstance(on_device(torch.device("cuda", 1)), torch.cuda.device)
    assert isinstance(on_device(torch.device("cuda", 0)), contextlib.nullcontext)
    assert isinstance(on_device(torch.device("cuda")), contextlib.nullcontext)


def test_gradients_of_the_norm_kernel_are_brought_to_the_grid():
    flat = torch.randn(1 + 8 * 16).to(BF)
    g = flat[1:].view(8, 16)
    assert g.data_ptr() % 16 and block.packed(None) is None
    p = block.packed(g)
    assert p.data_ptr() % 16 == 0 and p.is_contiguous() and torch.equal(p, g)
    t = torch.randn(16, 8).to(BF)
    assert block.packed(t) is t and torch.equal(block.packed(t.t()), t.t()) and block.packed(t.t()).is_contiguous()
