"""The hand-written tcgen05 / TMEM / TMA GEMM against a PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 256, 512), (256, 512, 1024), (1024, 1024, 1024),
                                    (2048, 3072, 1024), (4096, 1024, 4096), (8192, 2048, 1024)])
def test_gemm_matches_fp32_reference(m, n, k):
    from dfccl_b200.ops import gemm
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    c = gemm.matmul_nt(a, b)
    torch.cuda.synchronize()
    assert gemm.check_kernels()
    ref = a.float() @ b.float().t()
    err = (c.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, (err, scale)
    # the second call reuses tensor memory and barriers of a fresh launch
    c2 = gemm.matmul_nt(a, b)
    torch.cuda.synchronize()
    assert torch.equal(c, c2)


@pytest.mark.parametrize("a_t,b_t", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (256, 512, 192), (1024, 1024, 2048), (1536, 1024, 8192)])
def test_gemm_reads_transposed_operands_in_place(m, n, k, a_t, b_t):
    """Operands stored with the contraction index slow (A as [K, M], B as [K, N]) are described to the tensor cores as
    MN-major and read as they are: the data gradient (B transposed) and the weight gradient (both) of a linear layer."""
    from dfccl_b200.ops import gemm
    torch.manual_seed(m * 3 + n * 5 + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    a_in = a.t().contiguous() if a_t else a
    b_in = b.t().contiguous() if b_t else b
    c = gemm.matmul(a_in, b_in, a_transposed=a_t, b_transposed=b_t)
    torch.cuda.synchronize()
    assert gemm.check_kernels()
    ref = a.float() @ b.float().t()
    err = (c.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, (err, scale)
    assert torch.equal(c, gemm.matmul_nt(a, b))          # the same products in the same order: bit-identical to the K-major form


@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (512, 768, 448), (2048, 1024, 4096), (9728, 512, 1024)])
def test_cta_pair_kernel_agrees_with_the_one_cta_kernel(m, n, k, a_t, b_t, monkeypatch):
    """DFCCL_GEMM_PAIR=0 keeps products that would run on CTA pairs (cta_group::2) on a one-CTA form: here the last two (the
    first two run on one all the same).  Both accumulate the same products in the same order, so the results are
    bit-identical; 9728 rows = 38 row tiles x 2 column tiles make more tiles than resident pairs."""
    from dfccl_b200.ops import gemm
    torch.manual_seed(m + 7 * n + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    a_in = a.t().contiguous() if a_t else a
    b_in = b.t().contiguous() if b_t else b
    monkeypatch.setenv("DFCCL_GEMM_PAIR", "1")
    c_pair = gemm.matmul(a_in, b_in, a_transposed=a_t, b_transposed=b_t)
    torch.cuda.synchronize()
    assert gemm.check_kernels()
    monkeypatch.setenv("DFCCL_GEMM_PAIR", "0")
    c_one = gemm.matmul(a_in, b_in, a_transposed=a_t, b_transposed=b_t)
    torch.cuda.synchronize()
    ref = a.float() @ b.float().t()
    err = (c_pair.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, (err, scale)
    assert torch.equal(c_pair, c_one)


@pytest.mark.parametrize("m,n,k", [(8192, 4096, 64), (8192, 4096, 192), (2432, 4096, 256), (4864, 4096, 448), (2432, 2560, 1088), (4736, 4096, 576)])
def test_gemm_with_several_tiles_per_pair(m, n, k):
    """Two to seven tiles per pair, fewer and more steps of the contraction than there are stages: accumulators and stages are
    released only where somebody takes them again."""
    from dfccl_b200.ops import gemm
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    c = gemm.matmul_nt(a, b)
    again = [gemm.matmul_nt(a, b) for _ in range(4)]
    torch.cuda.synchronize()
    assert gemm.check_kernels()
    assert all(torch.equal(c, d) for d in again)
    ref = a.double() @ b.double().t()
    # one rounding to bf16 (8 significant bits: 2^-8 of the value at most) of an fp32 sum: k roundings of 2^-24 of partial sums below |a| |b|^T
    bound = ref.abs() * 2.0 ** -8 + (a.double().abs() @ b.double().abs().t()) * (k * 2.0 ** -24) + 1e-30
    assert bool(((c.double() - ref).abs() <= bound * 1.01).all())


def test_gemm_rejects_shapes_it_cannot_tile():
    from dfccl_b200.ops import gemm
    a = torch.randn(100, 64, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(256, 64, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(ValueError):
        gemm.matmul_nt(a, b)


def test_gemm_throughput_report():
    """Not an assertion on speed: prints achieved TFLOP/s next to cuBLAS for the record."""
    from dfccl_b200.ops import gemm
    m = n = k = 8192
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)

    def bench(fn):
        for _ in range(3):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(10):
            fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / 10

    import os
    os.environ["DFCCL_GEMM_PAIR"] = "0"
    one = bench(lambda: gemm.matmul_nt(a, b, out))
    os.environ["DFCCL_GEMM_PAIR"] = "1"
    ours = bench(lambda: gemm.matmul_nt(a, b, out))
    del os.environ["DFCCL_GEMM_PAIR"]
    cublas = bench(lambda: torch.matmul(a, b.t(), out=out))
    flops = 2.0 * m * n * k
    print(f"tcgen05 gemm 8192^3: CTA pairs {ours:.3f} ms = {flops / ours / 1e9:.0f} TFLOP/s; one CTA per tile {one:.3f} ms = "
          f"{flops / one / 1e9:.0f} TFLOP/s; cuBLAS {cublas:.3f} ms = {flops / cublas / 1e9:.0f} TFLOP/s")
    assert gemm.check_kernels()


@pytest.mark.parametrize("m,n,k", [
    (128, 512, 64), (128, 256, 192),                        # half a stage; a stage and a half
    (128, 256, 8256), (384, 256, 4160),                     # four slices of a contraction, of unequal length
    (256, 2048, 8192), (1024, 1024, 1024),                  # two slices; one narrow tile per SM
    (640, 2048, 4096), (896, 2304, 3072),                   # pairs of 256 x 128, the last row tile half empty
    (1280, 768, 1920), (1408, 2048, 1024),                  # pairs of 256 x 256, half empty
    (1920, 1280, 768), (2048, 1024, 448),
    (9600, 512, 1024), (9600, 1024, 192)])                  # persistent pairs, half empty
def test_every_tile_form_at_its_edges(m, n, k):
    """All storage orders give the same bits, and the error against 64 bits is that of one rounding to bf16: 2**-8 of a
    value at most, half of that in the 2-norm over many values (0.41 x 2**-8 = 2**-8 / sqrt(3) averaged over a binade)."""
    from dfccl_b200.ops import gemm
    torch.manual_seed(m + 3 * n + 5 * k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    out = torch.full((m + 128, n), 7.0, device="cuda", dtype=torch.bfloat16)       # rows behind the result stay as they are
    gemm.matmul_nt(a, b, out[:m])
    at, bt = a.t().contiguous(), b.t().contiguous()
    torch.cuda.synchronize()
    assert gemm.check_kernels()
    ref = a.double() @ b.double().t()
    assert ((out[:m].double() - ref).norm() / ref.norm()).item() < 2 ** -9
    assert bool((out[m:] == 7.0).all())
    for a_t, b_t in ((True, False), (False, True), (True, True)):
        assert torch.equal(out[:m], gemm.matmul(at if a_t else a, bt if b_t else b, a_transposed=a_t, b_transposed=b_t))


def test_chained_products_wait_for_one_another():
    """Launches overlap the set-up of the next product with the end of the one before: a chain in which every product
    reads the previous result (and overwrites what the one before it read) gives what separate launches give, in a
    stream and in a captured graph."""
    from dfccl_b200.ops import gemm
    torch.manual_seed(5)
    n = 512
    w = [(torch.randn(n, n, device="cuda") * n ** -0.5).to(torch.bfloat16) for _ in range(3)]
    x = torch.randn(256, n, device="cuda", dtype=torch.bfloat16)
    big = (torch.randn(256, 8192, device="cuda") * 0.02).to(torch.bfloat16)         # a longer kernel in front: 4 slices
    wb = (torch.randn(n, 8192, device="cuda") * 0.02).to(torch.bfloat16)
    h = [torch.empty(256, n, device="cuda", dtype=torch.bfloat16) for _ in range(2)]

    def chain(sync):
        gemm.matmul_nt(big, wb, h[0])
        h[0].add_(x)
        for i in range(12):
            gemm.matmul_nt(h[i % 2], w[i % 3], h[(i + 1) % 2])
            if sync:
                torch.cuda.synchronize()
        return h[0].clone()

    want = chain(True)
    for _ in range(5):
        assert torch.equal(chain(False), want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = chain(False)
    g.replay()
    torch.cuda.synchronize()
    assert gemm.check_kernels() and torch.equal(got, want)
