"""Tensor parallelism with sequence-parallel activations (Megatron style) on top of this library.

Forward passes run the fused kernels: the column-parallel layer is an all-gather -> GEMM, the
row-parallel layer a GEMM -> reduce-scatter, both one tcgen05 kernel each with the collective
inside (``dfccl_b200.ops.fused_linear``).  The data-gradient GEMMs of the backward passes are the same
two kernels with the roles swapped (the column-parallel layer's is a GEMM -> reduce-scatter, the
row-parallel layer's an all-gather -> GEMM, each on the transposed weight).  Biases, residuals and the GELU of an MLP ride in the products' epilogues
(on one rank; a pass over the operator's output on several).  On the host backend (tests) the layers
fall back to this library's stream-ordered collectives around plain GEMMs.

The reference has no tensor-parallel code; its simulator only generates the group structure of
such jobs (reference: simulator/simulator.py:434-493).
"""
from __future__ import annotations

from typing import Dict, Tuple

import torch
import torch.distributed as dist
import torch.nn as nn
from torch.autograd.function import once_differentiable

from .. import native as nv
from ..ops.block import BIAS, BIAS_GELU, BIAS_RES, GELU_GRAD, Epilogue, NO_EPILOGUE, apply_epilogue_, column_sum, epilogue_operand, packed, unhooked
from ..ops.fused_linear import AllGatherGemm, GemmReduceScatter, TpGroup
from ..utils.tensors import nccl_dtype, raw_stream


def _stream(t: torch.Tensor) -> int:
    return raw_stream(t.device) if t.device.type == "cuda" else 0


_OPS: Dict[Tuple, object] = {}


def shared_op(kind, tp: TpGroup, *shape):
    """Layers of the same shape share one fused operator (its heap buffers and rendezvous words):
    calls on one stream are ordered, and the operator's own done-handshake keeps a peer from
    overwriting what another still reads."""
    key = (kind.__name__, id(tp)) + tuple(shape)
    if key not in _OPS:
        _OPS[key] = kind(tp, *shape)
    return _OPS[key]


def _fused(tp: TpGroup) -> bool:
    """Fused kernels on GPUs; collective + plain GEMM on the host backend (tests) and on the comparison arm."""
    return tp.device.type == "cuda" and getattr(tp, "library", "dfccl") == "dfccl"


def _wgrad(gy: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """gy^T @ x (the weight gradient: a contraction over the token dimension).  Both operands are stored with the
    contraction index slow, which the tcgen05 kernel reads in place as MN-major operands; shapes it cannot tile go
    to ``torch.matmul``."""
    from ..ops import gemm
    if gy.is_cuda and gemm.gemm_supported(gy.shape[1], x.shape[1], gy.shape[0]):
        return gemm.matmul(gy, x, a_transposed=True, b_transposed=True)
    return gy.t() @ x


def tp_all_gather(tp: TpGroup, x: torch.Tensor) -> torch.Tensor:
    """Concatenate the ranks' tensors along dim 0 with this library's stream-ordered all-gather."""
    if tp.n == 1:
        return x
    x = x.contiguous()
    out = torch.empty((x.shape[0] * tp.n,) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device)
    if getattr(tp, "library", "dfccl") == "torch":         # comparison arm: the collective library behind torch.distributed
        dist.all_gather_into_tensor(out, x, group=tp.pg)
        return out
    nv.check(nv.lib().ncclAllGather(x.data_ptr(), out.data_ptr(), x.numel(), nccl_dtype(x.dtype), tp.comm.handle,
                                    _stream(x)), "ncclAllGather")
    return out


def tp_reduce_scatter(tp: TpGroup, x: torch.Tensor) -> torch.Tensor:
    """Sum over ranks, keep this rank's block of dim 0."""
    if tp.n == 1:
        return x
    x = x.contiguous()
    rows = x.shape[0] // tp.n
    out = torch.empty((rows,) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device)
    if getattr(tp, "library", "dfccl") == "torch":
        dist.reduce_scatter_tensor(out, x, group=tp.pg)
        return out
    nv.check(nv.lib().ncclReduceScatter(x.data_ptr(), out.data_ptr(), out.numel(), nccl_dtype(x.dtype), nv.SUM, tp.comm.handle,
                                        _stream(x)), "ncclReduceScatter")
    return out


class _ColumnFn(torch.autograd.Function):
    """y = all_gather(x_shard) W^T with plain GEMMs around this library's collectives (host backend, comparison arm).
    Backward: gW = gy^T x_full, gx_shard = reduce_scatter(gy W)."""

    @staticmethod
    def forward(ctx, x_shard, weight, layer):
        ctx.layer = layer
        ctx.save_for_backward(x_shard, weight)
        return tp_all_gather(layer.tp, x_shard) @ weight.t()

    @staticmethod
    def backward(ctx, gy):
        x_shard, weight = ctx.saved_tensors
        tp = ctx.layer.tp
        gy = gy.contiguous()
        x_full = tp_all_gather(tp, x_shard)
        return tp_reduce_scatter(tp, gy @ weight), gy.t() @ x_full, None


class _RowFn(torch.autograd.Function):
    """y_shard = reduce_scatter(x W^T), the same way.  Backward: gy = all_gather(gy_shard), gx = gy W, gW = gy^T x."""

    @staticmethod
    def forward(ctx, x, weight, layer):
        ctx.layer = layer
        ctx.save_for_backward(x, weight)
        return tp_reduce_scatter(layer.tp, x @ weight.t())

    @staticmethod
    def backward(ctx, gy_shard):
        x, weight = ctx.saved_tensors
        gy = tp_all_gather(ctx.layer.tp, gy_shard.contiguous())
        return gy @ weight, gy.t() @ x, None


# ---- on the fused kernels: bias, residual and GELU belong to the product.  One rank: in the GEMM's epilogue, and no
# ---- gathered copies; several ranks: one pass over the operator's output.
def _product(op, x: torch.Tensor, w: torch.Tensor, epi: Epilogue = NO_EPILOGUE, w_transposed: bool = False) -> torch.Tensor:
    if op.tp.n == 1:
        return op.local(x, w, w_transposed, epi)
    y = op(x, w, w_transposed=w_transposed)
    return apply_epilogue_(y, epi) if epi.kind else y


def _column(layer, x_shard: torch.Tensor, weight: torch.Tensor, epi: Epilogue):
    """(y, the gathered activations: what the weight gradient needs).  The operator's own buffer is shared by every layer
    of this shape, so several ranks keep a copy of it instead of gathering a second time in the backward pass."""
    x_shard = layer.op.operand(x_shard) if layer.tp.n == 1 else x_shard.contiguous()
    y = _product(layer.op, x_shard, weight, epi)
    return y, x_shard if layer.tp.n == 1 else layer.op.gathered.clone()


def _column_backward(layer, gy: torch.Tensor, x_full: torch.Tensor, weight: torch.Tensor):
    """gW, and the data gradient with the reduce-scatter inside the GEMM: gx = RS(gy [M, N/n] @ W [N/n, K]); the B operand is
    W^T, handed over as W itself (stored [contraction, output]: read in place as an MN-major operand)."""
    return _wgrad(gy, x_full), _product(layer.bwd_op, gy, weight, w_transposed=True)


def _row_backward(layer, gy_shard: torch.Tensor, x: torch.Tensor, weight: torch.Tensor, epi: Epilogue = NO_EPILOGUE):
    """gW, and the data gradient with the all-gather inside the GEMM, gx = AG(gy_shard) [M, N] @ W [N, K/n]; the operator's
    gathered buffer then holds the full output gradient, which gW needs."""
    gx = _product(layer.bwd_op, gy_shard, weight, epi, w_transposed=True)
    return _wgrad(gy_shard if layer.tp.n == 1 else layer.bwd_op.gathered, x), gx


def _bias_epilogue(bias, aux=None) -> Epilogue:
    if bias is None:
        return NO_EPILOGUE
    return Epilogue(BIAS, bias) if aux is None else Epilogue(BIAS_RES, bias, aux=aux)


class _ColumnFusedFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x_shard, weight, bias, layer):
        y, x_full = _column(layer, x_shard, weight, _bias_epilogue(bias))
        ctx.layer, ctx.has_bias = layer, bias is not None
        ctx.save_for_backward(x_full, weight)
        return y

    @staticmethod
    @once_differentiable
    def backward(ctx, gy):
        x_full, weight = ctx.saved_tensors
        gy = packed(gy)
        gb = column_sum(gy) if ctx.has_bias else None
        gw, gx = _column_backward(ctx.layer, gy, x_full, weight)
        return gx, gw, gb, None


class _RowFusedFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, residual, layer):
        x = layer.op.operand(x) if layer.tp.n == 1 else x.contiguous()
        ctx.layer, ctx.has_bias, ctx.has_residual = layer, bias is not None, residual is not None
        ctx.save_for_backward(x, weight)
        return _product(layer.op, x, weight, _bias_epilogue(bias, None if residual is None else residual.contiguous()))

    @staticmethod
    @once_differentiable
    def backward(ctx, gy_shard):
        x, weight = ctx.saved_tensors
        gy = packed(gy_shard)
        gb = column_sum(gy) if ctx.has_bias else None
        gw, gx = _row_backward(ctx.layer, gy, x, weight)
        return gx, gw, gb, gy_shard if ctx.has_residual else None, None


class _MlpFn(torch.autograd.Function):
    """residual + down(gelu(up(x))): GELU in the up product's epilogue, its gradient in the epilogue of down's data gradient."""

    @staticmethod
    def forward(ctx, x, up_weight, up_bias, down_weight, down_bias, residual, up, down):
        pre = torch.empty(up.op.m, up.op.n_out, dtype=torch.bfloat16, device=x.device) if any(ctx.needs_input_grad) else None
        act, x_full = _column(up, x, up_weight, Epilogue(BIAS_GELU, up_bias, pre=pre))
        ctx.up, ctx.down = up, down
        ctx.save_for_backward(x_full, pre, act, up_weight, down_weight)
        return _product(down.op, act, down_weight, Epilogue(BIAS_RES, down_bias, aux=residual.contiguous()))

    @staticmethod
    @once_differentiable
    def backward(ctx, gy_shard):
        x_full, pre, act, up_weight, down_weight = ctx.saved_tensors
        gy = packed(gy_shard)
        gb_down = column_sum(gy)
        gw_down, gpre = _row_backward(ctx.down, gy, act, down_weight, Epilogue(GELU_GRAD, aux=pre))
        gb_up = column_sum(gpre)
        gw_up, gx = _column_backward(ctx.up, gpre, x_full, up_weight)
        return gx, gw_up, gb_up, gw_down, gb_down, gy_shard, None, None


def _fused_bias(layer, x: torch.Tensor) -> bool:
    """The epilogues take bf16 activations and weights, and one bias per output feature."""
    return (x.dtype == layer.weight.dtype == torch.bfloat16 and layer.bias.is_contiguous()
            and epilogue_operand(layer.bias, (layer.op.n_out,), layer.weight.device))


def _fused_residual(layer, residual: torch.Tensor) -> bool:
    """And a residual of the output's own shape; anything that has to be cast or spread is added by torch."""
    return epilogue_operand(residual, (layer.op.rows, layer.op.n_out), layer.weight.device)


def gelu_mlp(up: "ColumnParallelLinear", down: "RowParallelLinear", x: torch.Tensor, residual: torch.Tensor) -> torch.Tensor:
    """``residual + down(gelu(up(x)))`` with the tanh form of GELU."""
    if (up.op is not None and down.op is not None and unhooked(up, ColumnParallelLinear) and unhooked(down, RowParallelLinear)
            and _fused_bias(up, x) and _fused_bias(down, x) and _fused_residual(down, residual)):
        return _MlpFn.apply(x, up.weight, up.bias, down.weight, down.bias, residual, up, down)
    return residual + down(nn.functional.gelu(up(x), approximate="tanh"))


class ColumnParallelLinear(nn.Module):
    """y[M, N/n] = all_gather(x_shard)[M, K] W_local^T + b_local.  Input is sequence-sharded, output is
    feature-sharded."""

    def __init__(self, tp: TpGroup, rows_per_rank: int, full_weight: torch.Tensor, parts: int = 1):
        """``full_weight`` [out, in] is the unsharded weight (identical on every rank); this rank keeps rows
        ``rank`` of each of its ``parts`` equal row groups (3 for a fused q/k/v projection)."""
        super().__init__()
        out_features, in_features = full_weight.shape
        assert out_features % (tp.n * parts) == 0
        self.tp = tp
        nl = out_features // tp.n
        w = full_weight.view(parts, tp.n, out_features // (parts * tp.n), in_features)[:, tp.rank]
        self.weight = nn.Parameter(w.reshape(nl, in_features).to(torch.bfloat16).contiguous())
        self.bias = nn.Parameter(torch.zeros(nl, dtype=torch.bfloat16, device=tp.device))
        self.op = shared_op(AllGatherGemm, tp, rows_per_rank, in_features, nl) if _fused(tp) else None
        self.bwd_op = shared_op(GemmReduceScatter, tp, rows_per_rank * tp.n, nl, in_features) if _fused(tp) else None

    def forward(self, x_shard):
        if self.op is None:
            return _ColumnFn.apply(x_shard, self.weight, self) + self.bias
        if _fused_bias(self, x_shard):
            return _ColumnFusedFn.apply(x_shard, self.weight, self.bias, self)
        return _ColumnFusedFn.apply(x_shard, self.weight, None, self) + self.bias


class RowParallelLinear(nn.Module):
    """y_shard[M/n, N] = reduce_scatter(x[M, K/n] W_local^T) + b.  Input is feature-sharded, output is
    sequence-sharded.  The bias is replicated (its gradient is summed over the group by the caller)."""

    def __init__(self, tp: TpGroup, m: int, full_weight: torch.Tensor):
        super().__init__()
        out_features, in_features = full_weight.shape
        assert in_features % tp.n == 0
        self.tp = tp
        kl = in_features // tp.n
        self.weight = nn.Parameter(full_weight[:, tp.rank * kl:(tp.rank + 1) * kl].to(torch.bfloat16).contiguous())
        self.bias = nn.Parameter(torch.zeros(out_features, dtype=torch.bfloat16, device=tp.device))
        self.bias.tp_replicated = True
        self.op = shared_op(GemmReduceScatter, tp, m, kl, out_features) if _fused(tp) else None
        self.bwd_op = shared_op(AllGatherGemm, tp, m // tp.n, out_features, kl) if _fused(tp) else None

    def forward(self, x, residual=None):
        """``residual`` (sharded like the output) is added in the same pass as the bias."""
        if self.op is not None and _fused_bias(self, x) and (residual is None or _fused_residual(self, residual)):
            return _RowFusedFn.apply(x, self.weight, self.bias, residual, self)
        y = (_RowFn.apply(x, self.weight, self) if self.op is None else _RowFusedFn.apply(x, self.weight, None, None, self)) + self.bias
        return y if residual is None else residual + y
