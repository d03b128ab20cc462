"""Layer surface: the ``mlx.nn`` modules PIE's Llama model instantiates, with the same constructor arguments,
parameter names (``weight`` / ``scales`` / ``biases``) and ``__call__`` semantics, over torch CUDA tensors.

Reference: MLX/python/mlx/nn/layers/quantized.py:11-229, normalization.py:142-143 (MLX = src/pie_core/external/mlx).
"""
from __future__ import annotations

import math

import torch

from . import ops


class Module:
    """Minimal stand-in for mlx.nn.Module: attribute tree + flat parameter dict with dotted names."""

    def children(self):
        for k, v in vars(self).items():
            if isinstance(v, Module):
                yield k, v
            elif isinstance(v, list) and v and isinstance(v[0], Module):
                for i, m in enumerate(v):
                    yield f"{k}.{i}", m

    def parameters(self, prefix: str = "") -> dict:
        out = {}
        for k, v in vars(self).items():
            if isinstance(v, torch.Tensor) and not k.startswith("_"):
                out[prefix + k] = v
        for k, m in self.children():
            out.update(m.parameters(prefix + k + "."))
        return out

    def load_weights(self, weights: dict, strict: bool = True):
        """nn.Module.load_weights: assign by dotted name; strict -> every parameter must be provided."""
        mine = self.parameters()
        if strict:
            missing = sorted(set(mine) - set(weights))
            extra = sorted(set(weights) - set(mine))
            if extra:
                raise ValueError(f"Received parameters not in model: {' '.join(extra[:8])}.")
            if missing:
                raise ValueError(f"Missing parameters: {' '.join(missing[:8])}.")
        for name, value in weights.items():
            if name not in mine:
                continue
            if tuple(value.shape) != tuple(mine[name].shape):
                raise ValueError(f"Expected shape {tuple(mine[name].shape)} but received shape "
                                 f"{tuple(value.shape)} for parameter {name}")
            obj = self
            parts = name.split(".")
            for p in parts[:-1]:
                obj = getattr(obj, p) if not p.isdigit() else obj[int(p)]
            setattr(obj, parts[-1], value)
        return self


class QuantizedLinear(Module):
    """nn.QuantizedLinear(input_dims, output_dims, bias, group_size, bits) (quantized.py:135-229).
    weight: uint32 words (held as int32) [output_dims, input_dims * bits / 32]; scales, biases: bf16
    [output_dims, input_dims / group_size]."""

    def __init__(self, input_dims: int, output_dims: int, bias: bool = True, group_size: int = 64, bits: int = 4,
                 device="cuda"):
        self.group_size, self.bits = group_size, bits
        scale = math.sqrt(1.0 / input_dims)
        w = (torch.rand((output_dims, input_dims), device=device) * 2 - 1) * scale
        self.weight, self.scales, self.biases = ops.quantize(w.to(torch.bfloat16), group_size, bits)
        if bias:
            self.bias = torch.zeros((output_dims,), dtype=torch.bfloat16, device=device)

    def __call__(self, x):
        if x.is_cuda and x.numel() <= 32 * x.shape[-1]:   # few rows: the bits of the call below, without its way through Python
            y = ops.native_fused_rows()(x, (self,), None, None, False, QuantizedLinear, RMSNorm, ops.qmv_workspace)
            if y is not None:
                return y
        y = ops.quantized_matmul(x, self.weight, self.scales, self.biases, transpose=True,
                                 group_size=self.group_size, bits=self.bits)
        if "bias" in vars(self):
            y = y + self.bias
        return y

    @classmethod
    def from_linear(cls, weight: torch.Tensor, bias=None, group_size: int = 64, bits: int = 4):
        out_dims, in_dims = weight.shape
        ql = cls.__new__(cls)
        ql.group_size, ql.bits = group_size, bits
        ql.weight, ql.scales, ql.biases = ops.quantize(weight, group_size, bits)
        if bias is not None:
            ql.bias = bias
        return ql


class QuantizedEmbedding(Module):
    """nn.QuantizedEmbedding(num_embeddings, dims, group_size, bits) (quantized.py:60-132)."""

    def __init__(self, num_embeddings: int, dims: int, group_size: int = 64, bits: int = 4, device="cuda"):
        self.group_size, self.bits = group_size, bits
        self.num_embeddings, self.dims = num_embeddings, dims
        w = torch.randn((num_embeddings, dims), device=device) * math.sqrt(1.0 / dims)
        self.weight, self.scales, self.biases = ops.quantize(w.to(torch.bfloat16), group_size, bits)

    def __call__(self, x):
        return ops.dequantize(self.weight, self.scales, self.biases, self.group_size, self.bits, ids=x)

    def as_linear(self, x):
        """Tied output head (quantized.py:109-124)."""
        return ops.quantized_matmul(x, self.weight, self.scales, self.biases, transpose=True,
                                    group_size=self.group_size, bits=self.bits)


def _plain(lin, bits: int, K: int) -> bool:
    """A bias-free QuantizedLinear whose arrays the kernels can take as they lie.  (Anything that can be called may stand in a
    layer's place: nothing of it is read before its type is known.)"""
    if type(lin) is not QuantizedLinear:
        return False
    w, s, b = lin.weight, lin.scales, lin.biases
    return not ("bias" in lin.__dict__ or lin.bits != bits or lin.group_size != 64
                or w.dtype != torch.int32 or w.dim() != 2 or w.shape[1] * 32 != K * bits or s.dtype != torch.bfloat16
                or b.dtype != torch.bfloat16 or s.shape != b.shape or s.shape != (w.shape[0], K // 64)
                or not (w.is_contiguous() and s.is_contiguous() and b.is_contiguous())
                or w.data_ptr() % 16 or s.data_ptr() % 8 or b.data_ptr() % 8)


def fused_swiglu(x, gate, up):
    """silu(gate(x)) * up(x) of a prompt's rows in ONE launch, rounding for rounding the separate calls.  None where that does not
    apply or does not pay (the caller then makes the separate calls, which also report what is wrong)."""
    K = x.shape[-1]
    if x.dtype != torch.bfloat16 or not x.is_contiguous() or K == 0 or x.numel() < 64 * K:
        return None
    if type(gate) is not QuantizedLinear or gate.bits not in (4, 8):
        return None
    if not ops.qmm_swiglu_pays(x.numel() // K, gate.weight.shape[0], K, gate.bits):
        return None
    if not _plain(gate, gate.bits, K) or not _plain(up, gate.bits, K) or gate.weight.shape != up.weight.shape:
        return None
    return ops.qmm_swiglu(x, gate, up, x.numel() // K, K)


def fused_prompt(x, linears, residual=None):
    """A prompt's rows (64 and more) through several bias-free QuantizedLinears in one launch, [..., sum N] their outputs side by side, and a
    residual added to them.  One matrix of more than 128 rows: the bits of the separate calls; several: theirs up to the order of fp32 sums over K, which
    may be cut in other places.  None where that does not apply (the caller then makes those)."""
    K = x.shape[-1]
    if x.dtype != torch.bfloat16 or not x.is_contiguous() or K == 0 or K % 128 or x.numel() < 64 * K:
        return None
    bits, N = getattr(linears[0], "bits", None), 0
    if bits not in (4, 8):
        return None
    for lin in linears:
        if not _plain(lin, bits, K):
            return None
        N += lin.weight.shape[0]
    if residual is not None and (residual.shape != x.shape[:-1] + (N,) or residual.dtype != torch.bfloat16 or not residual.is_contiguous()):
        return None
    return ops.qmm_rows(x, linears, x.numel() // K, K, N, residual)


def fused_rows(x, linears, norm=None, residual=None, swiglu: bool = False):
    """Up to 32 rows, and up to 128 where that is sooner done, through several bias-free QuantizedLinears in ONE pass over their weights, with
    the RMSNorm in front of them, and the residual sum or SwiGLU behind them where asked for:
        [..., sum N]  their outputs side by side;   residual: residual + output;   swiglu: silu(first) * second.
    Results are rounded where the separate calls round them.  One matrix, with or without a residual, gives their bits; a norm's
    sum of squares and the sums over K of several matrices are taken in another order, so that a value near a rounding boundary
    may fall on its other side.
    None where that kernel does not apply (the caller then makes the separate calls, which also report what is wrong)."""
    K = x.shape[-1]
    rows = x.numel() // K if K else 0
    if rows > 32:   # most such calls are the separate ones', and find out before anything else is looked at
        if rows > 128 or any(type(lin) is not QuantizedLinear for lin in linears):
            return None
        if not ops.qmt_scratch_bytes(rows, sum(lin.weight.shape[0] for lin in linears) // (2 if swiglu else 1), K, linears[0].bits, int(swiglu)):
            return None
    if x.is_cuda:
        y = ops.native_fused_rows()(x, linears, norm, residual, swiglu, QuantizedLinear, RMSNorm, ops.qmv_workspace)
        if y is not None:
            return y
    if not 0 < rows <= 128 or x.dtype != torch.bfloat16 or not x.is_contiguous() or x.data_ptr() % 16:
        return None
    bits, N = getattr(linears[0], "bits", None), 0
    if bits not in (4, 8) or K % (1024 // bits):
        return None
    for lin in linears:
        if not _plain(lin, bits, K):
            return None
        N += lin.weight.shape[0]
    if swiglu:
        if linears[0].weight.shape[0] != linears[1].weight.shape[0]:
            return None
        N //= 2
    if norm is not None:
        if type(norm) is not RMSNorm:
            return None
        nw = norm.weight
        if nw.dtype != torch.bfloat16 or nw.shape != (K,) or not nw.is_contiguous() or nw.data_ptr() % 16:
            return None
    if residual is not None and (residual.shape != x.shape[:-1] + (N,) or residual.dtype != torch.bfloat16
                                 or not residual.is_contiguous()):
        return None
    return ops.qmv_fused(x, linears, rows, K, N, bits, None if norm is None else norm.weight, 0.0 if norm is None else norm.eps,
                         residual, swiglu)


class RMSNorm(Module):
    """nn.RMSNorm(dims, eps) (normalization.py:105-143)."""

    def __init__(self, dims: int, eps: float = 1e-5, device="cuda"):
        self.weight = torch.ones((dims,), dtype=torch.bfloat16, device=device)
        self.eps = eps

    def __call__(self, x):
        return ops.rms_norm(x, self.weight, self.eps)
