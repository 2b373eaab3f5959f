"""The kernels around a transformer block's GEMMs against 64-bit torch: epilogues, layer norm, column sums, and a whole
block against the same block on torch's own operators."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
HALF_ULP = 2.0 ** -8                     # one rounding to bf16 (8 significant bits), relative, at most


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm().clamp_min(1e-300)).item()


# all on the persistent kernel (epilogue inside; 9600 rows: last row tile half empty) but 128 x 256 x 4096, whose contraction is cut:
# a tile form followed by a pass of its own
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (256, 768, 256), (8192, 1024, 1024), (9600, 512, 1024), (128, 256, 4096)])
def test_epilogues(native, m, n, k):
    from dfccl_b200.ops import block, gemm
    g = torch.Generator(device="cuda").manual_seed(m + n)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)              # noqa: E731
    a, b, bias, aux = rnd(m, k), (rnd(n, k) * k ** -0.5).to(torch.bfloat16), rnd(n), rnd(m, n)
    acc = a.double() @ b.double().t()
    pre, out = torch.empty_like(aux), torch.empty_like(aux)

    def run(epi):
        native.check(native.lib().dfcclGemmBf16Epilogue(a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, k, 0, 0, *epi.args(),
                                                        torch.cuda.current_stream().cuda_stream), "epilogue")
        return out.clone()

    gelu = lambda x: F.gelu(x, approximate="tanh")                                               # noqa: E731
    # a product rounded before its epilogue (a pass of its own) has one rounding more
    assert _rel(run(block.Epilogue(block.BIAS, bias)), acc + bias.double()) < 2 * HALF_ULP
    assert _rel(run(block.Epilogue(block.BIAS_RES, bias, aux=aux)), acc + bias.double() + aux.double()) < 2 * HALF_ULP
    y = run(block.Epilogue(block.BIAS_GELU, bias, pre=pre))
    assert _rel(pre, acc + bias.double()) < 2 * HALF_ULP
    assert _rel(y, gelu(pre.double())) < HALF_ULP
    assert torch.equal(run(block.Epilogue(block.BIAS_GELU, bias)), y)
    x = aux.double().requires_grad_(True)
    gelu(x).backward(acc)
    assert _rel(run(block.Epilogue(block.GELU_GRAD, aux=aux)), x.grad) < 2 * HALF_ULP
    torch.cuda.synchronize()
    assert gemm.check_kernels()


def test_gelu_far_from_zero(native):
    from dfccl_b200.ops import block
    v = torch.tensor([0.0, -0.0, 1e-30, 5.0, -5.0, 9.0, -9.0, -20.0, 3e4, -3e4, 1e12, -1e12, 3e38, -3e38, float("inf"), float("nan")],
                     device="cuda", dtype=torch.bfloat16).view(1, 16)
    y = block.apply_epilogue_(v.clone(), block.Epilogue(block.BIAS_GELU, torch.zeros(16, device="cuda", dtype=torch.bfloat16)))
    want = F.gelu(v.double(), approximate="tanh")
    # the reference's 1 + tanh is only good to 2**-53: times 20, the largest |x| at which the result is not 0
    assert torch.allclose(y.double()[:, :14], want[:, :14], rtol=2 * HALF_ULP, atol=20 * 2.0 ** -53)
    assert y[0, 14] == float("inf") and torch.isnan(y[0, 15])
    d = block.apply_epilogue_(torch.ones_like(v), block.Epilogue(block.GELU_GRAD, aux=v.clone()))
    x = v.double()[:, :12].clone().requires_grad_(True)
    F.gelu(x, approximate="tanh").sum().backward()
    assert torch.allclose(d.double()[:, :12], x.grad, rtol=2 * HALF_ULP, atol=1e-6)
    assert d[0, 12] == 1 and d[0, 13] == 0 and torch.isnan(d[0, 15])


@pytest.mark.parametrize("rows,d", [(1, 8), (3, 248), (37, 256), (130, 264), (1000, 768), (8192, 1024), (515, 1600), (64, 2048)])
def test_layer_norm_with_the_residuals_gradient(native, rows, d):
    from dfccl_b200.ops import block
    torch.manual_seed(rows + d)
    ln = nn.LayerNorm(d, dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        ln.weight.add_(torch.randn_like(ln.weight) * 0.1)
        ln.bias.add_(torch.randn_like(ln.bias) * 0.1)
    x = (torch.randn(rows, d, device="cuda") * 2 + 1).to(torch.bfloat16).requires_grad_(True)
    g1, g2 = (torch.randn(rows, d, device="cuda").to(torch.bfloat16) for _ in range(2))
    h, y = block.norm_residual(ln, x)
    torch.autograd.backward([h, y], [g1, g2])
    x64 = x.detach().double().requires_grad_(True)
    w64, b64 = ln.weight.detach().double().requires_grad_(True), ln.bias.detach().double().requires_grad_(True)
    y64 = F.layer_norm(x64, (d,), w64, b64, ln.eps)
    torch.autograd.backward([x64 * 1, y64], [g1.double(), g2.double()])
    assert torch.equal(h, x)
    # fp32 arithmetic (sums of up to 8192 terms), one rounding
    for got, want in ((y, y64), (x.grad, x64.grad), (ln.weight.grad, w64.grad), (ln.bias.grad, b64.grad)):
        assert _rel(got.detach(), want.detach()) < HALF_ULP


def test_layer_norm_with_gradients_off_the_grid(native):
    """Both gradients arrive as slices of a flat array, one element from its start."""
    from dfccl_b200.ops import block
    torch.manual_seed(8)
    ln = nn.LayerNorm(256, dtype=torch.bfloat16, device="cuda")
    x = torch.randn(37, 256, device="cuda").to(torch.bfloat16).requires_grad_(True)
    one = torch.zeros(1, device="cuda", dtype=torch.bfloat16)
    g1, g2 = (torch.randn(1 + x.numel(), device="cuda").to(torch.bfloat16) for _ in range(2))
    h, y = block.norm_residual(ln, x)
    torch.autograd.backward([torch.cat([one, h.reshape(-1)]), torch.cat([one, y.reshape(-1)])], [g1, g2])
    x64, w64, b64 = (t.detach().double().requires_grad_(True) for t in (x, ln.weight, ln.bias))
    torch.autograd.backward([x64 * 1, F.layer_norm(x64, (256,), w64, b64, ln.eps)], [g[1:].view(37, 256).double() for g in (g1, g2)])
    for got, want in ((x.grad, x64.grad), (ln.weight.grad, w64.grad), (ln.bias.grad, b64.grad)):
        assert _rel(got, want) < HALF_ULP


@pytest.mark.parametrize("rows,n", [(1, 8), (31, 64), (33, 264), (1000, 1024), (8192, 3072), (4100, 4096)])
def test_column_sum(native, rows, n):
    from dfccl_b200.ops import block
    torch.manual_seed(rows + n)
    g = torch.randn(rows, n, device="cuda").to(torch.bfloat16)
    assert _rel(block.column_sum(g), g.double().sum(0)) < HALF_ULP


@pytest.mark.parametrize("rows,n", [(16383, 200), (16384, 8), (16387, 200), (65536, 64), (65539, 264), (131072, 128), (16385, 1984), (16400, 2048)])
def test_column_sum_of_tall_matrices(native, rows, n):
    """In stretches of rows with scratch memory, and in one launch without."""
    from dfccl_b200.ops import block
    torch.manual_seed(rows + n)
    g = torch.randn(rows, n, device="cuda").to(torch.bfloat16)
    want, out = g.double().sum(0), torch.empty(n, device="cuda", dtype=torch.bfloat16)
    got = block.column_sum(g)
    assert _rel(got, want) < HALF_ULP
    assert torch.equal(got, block.column_sum(g))
    native.check(native.lib().dfcclColumnSum(g.data_ptr(), out.data_ptr(), None, rows, n, torch.cuda.current_stream().cuda_stream), "dfcclColumnSum")
    assert _rel(out, want) < HALF_ULP


@pytest.mark.parametrize("tokens,d,hooked", [(256, 256, False), (8192, 512, False), (256, 256, True)])
def test_block_against_torch_operators(native, tokens, d, hooked):
    """Output and every gradient of a one-rank block; modules with hooks are called as modules."""
    from dfccl_b200.models.gpt2 import GPT2Config, ParallelBlock
    from dfccl_b200.ops.fused_linear import TpGroup
    native.set_backend("cuda")
    (comm,) = native.Comm.init_loopback(1, 0)
    dev = torch.device("cuda", 0)
    cfg = GPT2Config(n_layer=1, d_model=d, n_head=d // 64, seq_len=128)
    blk = ParallelBlock(cfg, TpGroup(comm, None, dev), tokens, 0, 11)
    torch.manual_seed(3)
    with torch.no_grad():
        for p in blk.parameters():
            if p.dim() == 1:
                p.add_((torch.randn(p.shape, device=dev) * 0.1).to(p.dtype))
    calls = []
    if hooked:
        for m in (blk.ln1, blk.qkv, blk.proj, blk.ln2, blk.up, blk.down):
            m.register_forward_hook(lambda *_: calls.append(1))
    x = torch.randn(tokens, d, device=dev).to(torch.bfloat16).requires_grad_(True)
    gy = torch.randn(tokens, d, device=dev).to(torch.bfloat16)
    y = blk(x)
    y.backward(gy)
    assert len(calls) == (6 if hooked else 0)

    p = {k: v.detach().double().requires_grad_(True) for k, v in blk.named_parameters()}
    x64 = x.detach().double().requires_grad_(True)
    ln = lambda t, n: F.layer_norm(t, (d,), p[n + ".weight"], p[n + ".bias"])                     # noqa: E731
    lin = lambda t, n: t @ p[n + ".weight"].t() + p[n + ".bias"]                                  # noqa: E731
    q, k, v = (t.transpose(1, 2) for t in lin(ln(x64, "ln1"), "qkv").view(tokens // 128, 128, 3, d // 64, 64).unbind(2))
    a = F.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).reshape(tokens, d)
    h = x64 + lin(a, "proj")
    y64 = h + lin(F.gelu(lin(ln(h, "ln2"), "up"), approximate="tanh"), "down")
    y64.backward(gy.double())
    # bf16 activations through a whole block: a few roundings of 2**-8 at most each on the way to the output and back
    assert _rel(y.detach(), y64.detach()) < 1e-2 and _rel(x.grad, x64.grad) < 1e-2
    for name, q in blk.named_parameters():
        if name == "qkv.bias":                     # the key bias has no gradient but rounding noise (softmax is shift-invariant)
            keep = torch.cat([torch.arange(0, d), torch.arange(2 * d, 3 * d)]).to(dev)
            assert _rel(q.grad[keep], p[name].grad[keep]) < 2e-2, name
        else:
            assert _rel(q.grad, p[name].grad) < 2e-2, name
    comm.destroy()


@pytest.mark.parametrize("kind", ["ColumnParallelLinear", "RowParallelLinear"])
def test_layers_take_fp32_activations(native, kind):
    """An operator that is not registered with a context has always taken its input through a copy, which casts."""
    from dfccl_b200.ops.fused_linear import TpGroup
    from dfccl_b200.parallel import tp as tp_mod
    native.set_backend("cuda")
    (comm,) = native.Comm.init_loopback(1, 0)
    torch.manual_seed(5)
    w = torch.randn(512, 256, device="cuda") * 256 ** -0.5
    layer = getattr(tp_mod, kind)(TpGroup(comm, None, torch.device("cuda", 0)), 384, w)
    x = torch.randn(384, 256, device="cuda", requires_grad=True)
    gy = torch.randn(384, 512, device="cuda").to(torch.bfloat16)
    y = layer(x)
    y.backward(gy)
    x64, w64 = x.detach().to(torch.bfloat16).double().requires_grad_(True), layer.weight.detach().double().requires_grad_(True)
    (x64 @ w64.t()).backward(gy.double())
    # products of bf16 operands, summed in fp32, one rounding (the bias is zero: adding it rounds nothing)
    for got, want in ((y, x64 @ w64.t()), (x.grad, x64.grad), (layer.weight.grad, w64.grad)):
        assert _rel(got.detach(), want.detach()) < HALF_ULP
    assert x.grad.dtype == torch.float32
    comm.destroy()


@pytest.mark.parametrize("kind", ["ColumnParallelLinear", "RowParallelLinear"])
def test_layers_with_inputs_and_gradients_off_the_grid(native, kind):
    """Slices one element from the start of a flat array; the copy into an operand used to take them."""
    from dfccl_b200.ops.fused_linear import TpGroup
    from dfccl_b200.parallel import tp as tp_mod
    native.set_backend("cuda")
    (comm,) = native.Comm.init_loopback(1, 0)
    torch.manual_seed(9)
    layer = getattr(tp_mod, kind)(TpGroup(comm, None, torch.device("cuda", 0)), 256, torch.randn(512, 256, device="cuda") * 256 ** -0.5)
    flat = torch.randn(1 + 256 * 256, device="cuda").to(torch.bfloat16).requires_grad_(True)
    g = torch.randn(1 + 256 * 512, device="cuda").to(torch.bfloat16)
    y = layer(flat[1:].view(256, 256))
    torch.cat([g[:1], y.reshape(-1)]).backward(g)
    f64, w64, b64 = (t.detach().double().requires_grad_(True) for t in (flat, layer.weight, layer.bias))
    y64 = f64[1:].view(256, 256) @ w64.t() + b64
    y64.backward(g[1:].view(256, 512).double())
    for got, want in ((y, y64), (flat.grad, f64.grad), (layer.weight.grad, w64.grad), (layer.bias.grad, b64.grad)):
        assert _rel(got.detach(), want.detach()) < HALF_ULP
    comm.destroy()


@pytest.mark.parametrize("residual", ["same", "strided", "row", "vector", "column", "misaligned", "fp32"])
@pytest.mark.parametrize("bias", ["full", "misaligned", "one"])
def test_residuals_and_biases_of_any_form(native, residual, bias):
    """What the epilogue takes as it is and what is added by torch, with gradients."""
    from dfccl_b200.ops.fused_linear import TpGroup
    from dfccl_b200.parallel.tp import RowParallelLinear
    native.set_backend("cuda")
    (comm,) = native.Comm.init_loopback(1, 0)
    torch.manual_seed(6)
    m, n, k = 256, 512, 256
    rnd = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)                           # noqa: E731
    layer = RowParallelLinear(TpGroup(comm, None, torch.device("cuda", 0)), m, torch.randn(n, k, device="cuda") * k ** -0.5)
    layer.bias = nn.Parameter({"full": lambda: rnd(n), "misaligned": lambda: rnd(n + 1)[1:], "one": lambda: rnd(1)}[bias]())
    r = {"same": lambda: rnd(m, n), "strided": lambda: rnd(n, m).t(), "row": lambda: rnd(1, n), "vector": lambda: rnd(n), "column": lambda: rnd(m, 1),
         "misaligned": lambda: rnd(m * n + 1)[1:].view(m, n), "fp32": lambda: torch.randn(m, n, device="cuda")}[residual]().requires_grad_(True)
    x, gy = rnd(m, k).requires_grad_(True), rnd(m, n)
    y = layer(x, r)
    y.backward(gy.to(y.dtype))
    leaves = [t.detach().double().requires_grad_(True) for t in (x, layer.weight, layer.bias, r)]
    y64 = leaves[0] @ leaves[1].t() + leaves[2] + leaves[3]
    y64.backward(gy.double())
    # three roundings to bf16 where bias and residual are added one by one; gradients are sums rounded once
    assert y.dtype == (r.dtype if residual == "fp32" else torch.bfloat16) and _rel(y.detach(), y64.detach()) < 3 * HALF_ULP
    for got, want in zip((x, layer.weight, layer.bias, r), leaves):
        assert _rel(got.grad, want.grad) < 2 * HALF_ULP
    comm.destroy()


@pytest.mark.multigpu
def test_a_second_device_of_the_process(native):
    """Shared-memory limits are set on every device a kernel is launched on: widths above 768 (layer norm backward), tile
    forms and the persistent kernel, on device 1 after device 0."""
    from dfccl_b200.ops import block, gemm
    for dev in (0, 1):
        with torch.cuda.device(dev):
            ln = nn.LayerNorm(1024, dtype=torch.bfloat16, device=f"cuda:{dev}")
            x = torch.randn(512, 1024, device=f"cuda:{dev}").to(torch.bfloat16).requires_grad_(True)
            block.norm_residual(ln, x)[1].sum().backward()
            assert bool(torch.isfinite(x.grad).all())
            for m in (128, 8192):
                a = torch.ones(m, 1024, device=f"cuda:{dev}", dtype=torch.bfloat16)
                assert bool((gemm.matmul_nt(a, torch.ones_like(a[0]).expand(1024, 1024).contiguous()) == 1024).all())


@pytest.mark.multigpu
def test_tensors_of_a_device_that_is_not_current(native):
    from dfccl_b200.ops import block
    with torch.cuda.device(0):
        ln = nn.LayerNorm(256, dtype=torch.bfloat16, device="cuda:1")
        x = torch.randn(64, 256, device="cuda:1").to(torch.bfloat16).requires_grad_(True)
        h, y = block.norm_residual(ln, x)
        (h + y).float().square().sum().backward()
        assert bool(torch.isfinite(x.grad).all())
        assert _rel(block.column_sum(x.detach()), x.detach().double().sum(0)) < HALF_ULP
        block.apply_epilogue_(torch.zeros_like(x.detach()), block.Epilogue(block.BIAS, ln.weight.detach()))
        torch.cuda.synchronize(1)
        assert torch.cuda.current_device() == 0


@pytest.mark.parametrize("adamw", [False, True])
def test_one_optimizer_launch_over_many_buckets(native, adamw):
    """More buckets than a launch holds, of both parameter types and odd lengths, against one call per bucket: the same
    bits, gradients cleared, nothing behind a bucket's end touched."""
    native.set_backend("cuda")
    L, st = native.lib(), torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(4)
    sizes = [1, 3, 4, 7, 2047, 2048, 2049, 100003, 0, 8, 4096, 5, 6, 1 << 20, 12, 16, 20, 2050]
    pad = 8
    rows, want = [], []
    for i, n in enumerate(sizes):
        ptype = torch.bfloat16 if i % 3 else torch.float32
        f = [torch.rand(n + pad, device="cuda", generator=gen) for _ in range(4)]
        p, c = torch.full((n + pad,), 3.0, device="cuda", dtype=ptype), torch.full((n + pad,), 5.0, device="cuda", dtype=ptype)
        rows.append((n, *f, p, c))
        want.append([t.clone() for t in (f[0], f[2], f[3], p)])
    for (n, _, g, *_, p, _), (w, m, v, q) in zip(rows, want):
        a = (w.data_ptr(), g.data_ptr(), m.data_ptr())
        t = native.BFLOAT16 if p.dtype == torch.bfloat16 else native.FLOAT32
        if adamw:
            native.check(L.dfcclFusedAdamWStep(*a, v.data_ptr(), q.data_ptr(), n, t, 0.01, 0.9, 0.99, 1e-8, 0.1, 2, st), "one")
        else:
            native.check(L.dfcclFusedSgdStep(*a, q.data_ptr(), n, t, 0.1, 0.9, 0.01, 0, st), "one")
    arr = (native.OptimBucket * len(rows))()
    for k, (n, w, g, m, v, p, c) in zip(arr, rows):
        k.master, k.grad32, k.momentum, k.moment2, k.param, k.clear = (t.data_ptr() for t in (w, g, m, v, p, c))
        k.n, k.param_type = n, native.BFLOAT16 if p.dtype == torch.bfloat16 else native.FLOAT32
    if adamw:
        native.check(L.dfcclFusedAdamWSteps(arr, len(rows), 0.01, 0.9, 0.99, 1e-8, 0.1, 2, st), "all")
    else:
        native.check(L.dfcclFusedSgdSteps(arr, len(rows), 0.1, 0.9, 0.01, 0, st), "all")
    for (n, w, g, m, v, p, c), ref in zip(rows, want):
        assert all(torch.equal(x, y) for x, y in zip((w, m, v, p), ref))
        assert bool((p[n:] == 3).all()) and bool((c[:n] == 0).all()) and bool((c[n:] == 5).all())
