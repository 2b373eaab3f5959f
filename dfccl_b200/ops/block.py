"""Kernels around the GEMMs of a transformer block (``csrc/src/ops/block.cu``): layer norm with the residual's gradient,
column sums (bias gradients), and what a GEMM does with its product before storing it (``csrc/src/gemm/epilogue.h``)."""
from __future__ import annotations

import functools
from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn as nn
from torch.autograd.function import once_differentiable

from .. import native as nv
from ..utils.tensors import on_device, raw_stream, stream_of

NONE, BIAS, BIAS_RES, BIAS_GELU, GELU_GRAD = range(5)


@dataclass
class Epilogue:
    """BIAS: ``+ bias``; BIAS_RES: ``+ bias + aux``; BIAS_GELU: ``pre = product + bias`` (stored if given), ``gelu(pre)``;
    GELU_GRAD: ``product * gelu'(aux)``.  bf16 tensors; ``aux`` and ``pre`` have the product's shape."""
    kind: int = NONE
    bias: Optional[torch.Tensor] = None
    aux: Optional[torch.Tensor] = None
    pre: Optional[torch.Tensor] = None

    def args(self):
        for t in (self.bias, self.aux, self.pre):
            assert t is None or (t.dtype == torch.bfloat16 and t.is_cuda and t.is_contiguous())
        return self.kind, _ptr(self.bias), _ptr(self.aux), _ptr(self.pre)

    def args_for(self, m: int, n: int):
        """The same for a product of [m, n]; the kernels read and write by address alone."""
        for t, shape in ((self.bias, (n,)), (self.aux, (m, n)), (self.pre, (m, n))):
            if t is not None and t.shape != shape:
                raise ValueError(f"operand of {tuple(t.shape)} in the epilogue of a product of {m} x {n}")
        return self.args()


def epilogue_operand(t: Optional[torch.Tensor], shape, device: torch.device) -> bool:
    """True if a bias or residual can ride in an epilogue: bf16 of just this shape, on this device, 16-byte aligned."""
    return (t is not None and t.dtype == torch.bfloat16 and tuple(t.shape) == tuple(shape) and t.device == device
            and (not t.is_contiguous() or t.data_ptr() % 16 == 0))


NO_EPILOGUE = Epilogue()


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def packed(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """Contiguous and 16-byte aligned (a gradient may be a slice of anything)."""
    if t is None:
        return None
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def apply_epilogue_(product: torch.Tensor, epi: Epilogue) -> torch.Tensor:
    """In place, for products whose kernel has no epilogue."""
    assert product.dtype == torch.bfloat16 and product.dim() == 2 and product.is_contiguous()
    m, n = product.shape
    args = epi.args_for(m, n)
    with on_device(product.device):
        nv.check(nv.lib().dfcclApplyEpilogue(product.data_ptr(), m, n, *args, raw_stream(product.device)), "dfcclApplyEpilogue")
    return product


@functools.lru_cache(maxsize=1024)
def _work_words(entry: str, device: int, rows: int, n: int) -> int:
    """fp32 words of scratch memory: a function of the sizes and of the device, which is the current one."""
    return getattr(nv.lib(), entry)(rows, n)


@functools.lru_cache(maxsize=1)
def _max_width() -> int:
    return nv.lib().dfcclLayerNormMaxWidth()


def column_sum(g: torch.Tensor) -> torch.Tensor:
    """Sum over the rows of a contiguous bf16 matrix, in fp32, rounded once."""
    rows, n = g.shape
    out = torch.empty(n, dtype=torch.bfloat16, device=g.device)
    with on_device(g.device):
        words = _work_words("dfcclColumnSumWork", g.get_device(), rows, n)
        work = torch.empty(words, dtype=torch.float32, device=g.device) if words else None
        nv.check(nv.entry("dfcclColumnSum")(g.data_ptr(), out.data_ptr(), _ptr(work), rows, n, stream_of(g)), "dfcclColumnSum")
    return out


class _NormFn(torch.autograd.Function):
    """(x, layer_norm(x)): the first output passes x on to the residual connection, so that its gradient is added by the
    norm's own backward kernel."""

    @staticmethod
    def forward(ctx, x, gamma, beta, eps):
        rows, d = x.shape
        y = torch.empty_like(x)
        stats = torch.empty(2, rows, dtype=torch.float32, device=x.device)
        with on_device(x.device):
            mean = stats.data_ptr()
            nv.check(nv.lib().dfcclLayerNormForward(x.data_ptr(), gamma.data_ptr(), beta.data_ptr(), y.data_ptr(), mean, mean + 4 * rows,
                                                    rows, d, eps, stream_of(x)), "dfcclLayerNormForward")
        ctx.save_for_backward(x, gamma, stats)
        ctx.set_materialize_grads(False)
        return x, y

    @staticmethod
    @once_differentiable
    def backward(ctx, gpass, gy):
        x, gamma, stats = ctx.saved_tensors
        if gy is None:
            return gpass, None, None, None
        rows, d = x.shape
        gy, gpass = packed(gy), packed(gpass)
        gx, gg, gb = torch.empty_like(x), torch.empty_like(gamma), torch.empty_like(gamma)
        with on_device(x.device):
            work = torch.empty(_work_words("dfcclLayerNormWork", x.get_device(), rows, d), dtype=torch.float32, device=x.device)
            mean = stats.data_ptr()
            nv.check(nv.entry("dfcclLayerNormBackward")(gy.data_ptr(), x.data_ptr(), gamma.data_ptr(), mean, mean + 4 * stats.stride(0), _ptr(gpass),
                                                        gx.data_ptr(), gg.data_ptr(), gb.data_ptr(), work.data_ptr(), rows, d, stream_of(x)),
                     "dfcclLayerNormBackward")
        return gx, gg, gb, None


def unhooked(m: nn.Module, cls: type) -> bool:
    """True if calling ``m`` does nothing but its class's forward, so that a fused form may stand in for the call."""
    return (type(m) is cls and "forward" not in m.__dict__ and not m._forward_hooks and not m._forward_pre_hooks
            and not m._backward_hooks and not m._backward_pre_hooks and not nn.modules.module._has_any_global_hook())


def norm_residual(ln: nn.LayerNorm, x: torch.Tensor):
    """``(x, ln(x))``.  The hand-written kernels for contiguous bf16 rows on a GPU (widths a multiple of 8 up to the
    kernels' limit); anything else goes through the module."""
    ok = (unhooked(ln, nn.LayerNorm) and x.is_cuda and x.dim() == 2 and x.dtype == torch.bfloat16 and x.is_contiguous() and x.shape[0] > 0
          and tuple(ln.normalized_shape) == (x.shape[1],) and x.shape[1] % 8 == 0 and x.shape[1] <= _max_width()
          and all(p is not None and p.dtype == torch.bfloat16 and p.device == x.device and p.is_contiguous() and p.data_ptr() % 16 == 0
                  for p in (ln.weight, ln.bias))
          and x.data_ptr() % 16 == 0 and not torch.is_autocast_enabled("cuda"))
    return _NormFn.apply(x, ln.weight, ln.bias, ln.eps) if ok else (x, ln(x))
