"""Persistent tiles of 256 x width: widths that cut the last column tile, an MN-major operand whose blocks of 64 columns the tiles
cut through, odd numbers of 64-wide contraction blocks, a half empty last row tile, more tiles than pairs and fewer; the tile form of
256 x 256 at the edges of its range."""
import pytest
import torch

from test_dispatch_rules import gemm_plan

pytestmark = pytest.mark.gpu

# (m, n, k), width with B stored K-major and MN-major (0: a tile form runs it; T: the one of 256 x 256)
T = "tile"
SHAPES = [((512, 1280, 2304), 64, 0), ((1408, 512, 2368), 64, 0),
          ((128, 4864, 3840), 96, 0), ((2432, 512, 4544), 96, 0),                         # the last tile 64 columns
          ((6528, 1024, 2496), 128, 128), ((2560, 2816, 1728), 224, 128),
          ((2432, 1024, 256), 160, 160), ((4096, 1280, 2368), 160, 160),                  # the last tile 64 columns / whole tiles
          ((2816, 1792, 2240), 160, 160),                                                 # 32 columns
          ((4864, 512, 256), 192, 192), ((1536, 2304, 320), 192, 192),
          ((3072, 1024, 2112), 224, 192), ((1152, 5632, 512), 224, 224), ((2688, 2560, 320), 224, 224),        # 128, 32, 96 columns
          ((384, 7936, 256), 256, 256), ((896, 4096, 256), 256, 256), ((2304, 3584, 576), 256, 256),
          ((1152, 3328, 2624), T, T), ((640, 5120, 512), T, T), ((4096, 1024, 576), T, T)]


@pytest.mark.parametrize("shape,k_major,mn_major", SHAPES)
def test_widths_at_their_edges(shape, k_major, mn_major):
    """The error against 64 bits is that of one rounding to bf16 (2**-8 of a value at most, 2**-9 in the 2-norm over many), the
    same bits for every storage order, and nothing outside the result is written."""
    from dfccl_b200.ops import gemm
    m, n, k = shape
    for b_t, want in ((False, k_major), (True, mn_major)):
        _, tile, _, width = gemm_plan(m, n, k, b_t)
        assert (tile == 256) if want == T else width == want
    torch.manual_seed(m + 3 * n + 5 * k)
    a = torch.randn(m, k, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(n, k, device="cuda", dtype=torch.bfloat16)
    out = torch.full((m + 128, n), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm.matmul_nt(a, b, out[:m])
    torch.cuda.synchronize()
    assert gemm.check_kernels()
    ref = a.double() @ b.double().t()
    assert ((out[:m].double() - ref).norm() / ref.norm()).item() < 2 ** -9
    assert bool((out[m:] == 7.0).all())
    at, bt = a.t().contiguous(), b.t().contiguous()
    for a_t, b_t in ((True, False), (False, True), (True, True)):
        assert torch.equal(out[:m], gemm.matmul(at if a_t else a, bt if b_t else b, a_transposed=a_t, b_transposed=b_t))
    assert gemm.check_kernels()


@pytest.mark.parametrize("m,n,k", [(1024, 768, 256), (128, 256, 64), (2176, 2304, 2048), (1408, 1024, 320)])
def test_epilogues_inside_ragged_tiles(m, n, k):
    """Small products with an epilogue run on the persistent kernel too: one rounding, for every kind."""
    from dfccl_b200 import native as nv
    from dfccl_b200.ops import block
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    b = (torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16)
    bias, aux = torch.randn(n, device="cuda").to(torch.bfloat16), torch.randn(m, n, device="cuda").to(torch.bfloat16)
    acc = a.double() @ b.double().t()
    x = aux.double().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").sum().backward()
    pre = torch.empty_like(aux)
    want = {block.BIAS: acc + bias.double(), block.BIAS_RES: acc + bias.double() + aux.double(), block.GELU_GRAD: acc * x.grad}
    for kind in (block.BIAS, block.BIAS_RES, block.GELU_GRAD, block.BIAS_GELU):
        epi = block.Epilogue(kind, bias if kind != block.GELU_GRAD else None, aux if kind in (block.BIAS_RES, block.GELU_GRAD) else None,
                             pre if kind == block.BIAS_GELU else None)
        out = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
        nv.check(nv.lib().dfcclGemmBf16Epilogue(a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, k, 0, 0, *epi.args(),
                                                torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        if kind == block.BIAS_GELU:                # of the rounded value, which is stored too: two roundings
            ref = acc + bias.double()
            assert ((pre.double() - ref).norm() / ref.norm()).item() < 2 ** -9
            ref = torch.nn.functional.gelu(pre.double(), approximate="tanh")
        else:
            ref = want[kind]
        assert ((out.double() - ref).norm() / ref.norm()).item() < 2 ** -9


@pytest.mark.parametrize("m,n,k", [(4096, 3072, 704), (4096, 3072, 768), (4096, 3072, 1024), (3840, 1792, 960), (2176, 2304, 704), (2176, 2304, 832)])
def test_bias_on_either_side_of_the_line(m, n, k):
    """Several tiles per pair, results through boxes and straight from the registers: one rounding, nothing behind the result."""
    from dfccl_b200 import native as nv
    from dfccl_b200.ops import block
    assert gemm_plan(m, n, k, False, 1)[3] >= 160
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    b = (torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda").to(torch.bfloat16)
    out = torch.full((m + 128, n), 7.0, device="cuda", dtype=torch.bfloat16)
    nv.check(nv.lib().dfcclGemmBf16Epilogue(a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, k, 0, 0, *block.Epilogue(block.BIAS, bias).args(),
                                            torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    ref = a.double() @ b.double().t() + bias.double()
    assert ((out[:m].double() - ref).norm() / ref.norm()).item() < 2 ** -9
    assert bool((out[m:] == 7.0).all())
