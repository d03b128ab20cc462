"""Operator surface of the path, with the names, argument meaning and error behaviour of the MLX operators
PIE's Llama model reaches: ``quantize``, ``dequantize``, ``quantized_matmul``, ``rms_norm``,
``rope``, ``scaled_dot_product_attention``.  Tensors are torch CUDA tensors; activations, scales, biases and
norm weights are bf16; packed weights are MLX ``uint32`` words held as ``torch.int32`` (same bits).

Every function is one or two calls into libpie_b200.so on the current CUDA stream.  No CPU fallback.
"""
from __future__ import annotations

import ctypes as C
import functools
import importlib.util
import os
import threading
import warnings

import torch

from . import _lib
from ._lib import EPI_RESADD, EPI_SILUMUL, EPI_STORE, HeadRows, KvLayout, KvqCache, QmvSeg

_BF16 = torch.bfloat16


def _p(t):
    return None if t is None else t.data_ptr()


def _stream():
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


@functools.lru_cache(maxsize=4096)
def _qmv_workspace_bytes(M: int, N: int, K: int, bits: int, dual: int) -> int:
    """A pure function of the sizes, asked for at every call."""
    return _lib.load().pie_qmv_workspace_bytes(M, N, K, bits, dual, 0)


def qmt_scratch_bytes(M: int, N: int, K: int, bits: int, dual: int) -> int:
    """0: the call is not for pie_qmt.  (Asked each time: it is the current device's answer.)"""
    return _lib.load().pie_qmt_scratch_bytes(M, N, K, 64, bits, dual) if 0 < M <= 128 else 0


def _qmt(out, x, segs, nseg, M: int, K: int, N: int, bits: int, norm_weight, eps, epilogue, residual, dual: int) -> bool:
    """pie_qmt where it serves the call.  Its scratch lives until the launch is queued and is reused in stream order, as any tensor."""
    nb = qmt_scratch_bytes(M, N, K, bits, dual)
    if not nb:
        return False
    scratch = torch.empty(nb, dtype=torch.uint8, device=x.device)
    status = _lib.load().pie_qmt(_p(out), N, _p(x), K, M, K, segs, nseg, 64, bits, _p(norm_weight), eps, epilogue, _p(residual),
                                 _p(scratch), nb, _stream())
    if status == _lib.EUNSUPPORTED:
        return False
    _lib.check(status, "qmt")
    return True


def _as_words(w: torch.Tensor) -> torch.Tensor:
    if w.dtype == torch.int32:
        return w
    if w.dtype == torch.uint32:
        return w.view(torch.int32)
    raise ValueError(f"[quantized_matmul] The weight matrix should be uint32 but received {w.dtype}")


def _check_gs_bits(what, group_size, bits, full=False):
    # MLX/mlx/fast.cpp:839-866
    if group_size not in (32, 64, 128):
        raise ValueError(f"[{what}] The requested group size {group_size} is not supported. "
                         "The supported group sizes are 32, 64 and 128.")
    if bits not in (2, 3, 4, 6, 8):
        raise ValueError(f"[{what}] The requested number of bits {bits} is not supported. "
                         "The supported bits are 2, 3, 4, 6 and 8.")
    if bits in (3, 6) or (full and (group_size != 64 or bits not in (4, 8))):
        raise ValueError(f"[{what}] group_size={group_size}, bits={bits} is valid MLX but not built for sm_100a here "
                         "(supported: group_size 64, bits 4 or 8)")


_raw_stream = torch._C._cuda_getCurrentRawStream
_capturing = torch.cuda.is_current_stream_capturing


def _capture_id() -> int:
    """Which capture into a graph the current stream is in."""
    return _lib.load().pie_capture_id(_stream())


class _Mine(threading.local):
    """A thread's workspaces: {(key, device, stream): buffer}, and those of the capture it is in."""

    def __init__(self):
        self.eager, self.captured, self.capture = {}, {}, 0


class _Workspaces:
    """Zero-initialised scratch owned by the host side (the library never allocates).

    A launch leaves its counters at zero for the next one in its buffer, so a buffer is for launches that come one after the other: one thread's, on one stream.  In a
    capture the buffers are the graph's, zeroed as part of it and kept for as long as the capture goes on: an eager call never sees one, and no graph holds the address of an
    eager call's, which is given back when a larger one is asked for.  A thread keeps the last KEEP of them, and gives them back when it ends."""

    KEEP = 96   # (a decode step's attention has one per 64 rows x query heads)

    def __init__(self):
        self.mine = _Mine()

    def get(self, key, nbytes, device):
        mine, index = self.mine, device.index
        stream = _raw_stream(index)
        bufs = mine.eager
        if stream and _capturing():   # (asking costs what the rest of this does, and the default stream cannot be captured)
            capture = _capture_id()
            if capture != mine.capture:
                mine.capture, mine.captured = capture, {}
            bufs = mine.captured
        elif mine.captured:           # that capture has ended, or this is another stream
            mine.capture, mine.captured = 0, {}
        key = (key, index, stream)
        buf = bufs.get(key)
        if buf is None or buf.numel() < nbytes:
            bufs.pop(key, None)
            buf = bufs[key] = torch.zeros(max(int(nbytes), 256), dtype=torch.uint8, device=device)
            if len(bufs) > self.KEEP:
                del bufs[next(iter(bufs))]   # the oldest; its memory is used again in its stream's order
        return buf


workspaces = _Workspaces()


def qmv_workspace(nbytes: int, device) -> torch.Tensor:
    return workspaces.get("qmv", nbytes, device)


def quantize(w: torch.Tensor, group_size: int = 64, bits: int = 4):
    """mx.quantize (MLX/mlx/ops.cpp:4023-4029; cpu/quantized.cpp:603-661).  Bit-exact with the reference."""
    _check_gs_bits("quantize", group_size, bits)
    if w.dim() < 2:
        raise ValueError("[quantize] The matrix to be quantized must have at least 2 dimension but it has only "
                         f"{w.dim()}.")
    if w.shape[-1] % group_size != 0:
        raise ValueError("[quantize] The last dimension of the matrix needs to be divisible by the quantization "
                         f"group size {group_size}. However the provided matrix has shape {tuple(w.shape)}")
    if w.dtype not in (_BF16, torch.float32):
        raise ValueError(f"[quantize] dtype {w.dtype} not built here (bfloat16 / float32)")
    w = w.contiguous()
    K = w.shape[-1]
    rows = w.numel() // K
    wq = torch.empty(w.shape[:-1] + (K * bits // 32,), dtype=torch.int32, device=w.device)
    s = torch.empty(w.shape[:-1] + (K // group_size,), dtype=w.dtype, device=w.device)
    b = torch.empty_like(s)
    L = _lib.load()
    _lib.check(L.pie_quantize(_p(w), 0 if w.dtype == _BF16 else 1, _p(wq), _p(s), _p(b), rows, K, group_size, bits,
                              _stream()), "quantize")
    return wq, s, b


def dequantize(w, scales, biases, group_size: int = 64, bits: int = 4, ids: torch.Tensor | None = None):
    """mx.dequantize (MLX/mlx/fast.cpp:917-1029), optionally gathering rows ``ids`` first
    (QuantizedEmbedding.__call__, MLX/python/mlx/nn/layers/quantized.py:100-107)."""
    _check_gs_bits("dequantize", group_size, bits)
    w = _as_words(w)
    if w.dim() < 2 or scales.dim() < 2 or biases.dim() < 2:
        raise ValueError("[dequantize] The matrix to be quantized must have at least 2 dimension.")
    if scales.shape != biases.shape:
        raise ValueError("[dequantize] Shape of scales and biases does not match")
    if w.shape[-1] * 32 // bits != scales.shape[-1] * group_size:
        raise ValueError(f"[dequantize] Shape of scales and biases does not match the matrix given the quantization "
                         f"parameters. Provided matrix of shape {tuple(w.shape)} and scales/biases of shape "
                         f"{tuple(scales.shape)} with group_size={group_size} and bits={bits}.")
    if scales.dtype != _BF16:
        raise ValueError("[dequantize] only bfloat16 scales/biases are built here")
    w, scales, biases = w.contiguous(), scales.contiguous(), biases.contiguous()
    K = w.shape[-1] * 32 // bits
    table_rows = w.numel() // w.shape[-1]
    if ids is None:
        out_shape, n_rows, idp = w.shape[:-1] + (K,), table_rows, None
    else:
        ids = ids.to(torch.int32).contiguous()
        out_shape, n_rows, idp = tuple(ids.shape) + (K,), ids.numel(), _p(ids)
    out = torch.empty(out_shape, dtype=_BF16, device=w.device)
    L = _lib.load()
    _lib.check(L.pie_dequantize(_p(out), _p(w), _p(scales), _p(biases), idp, n_rows, table_rows, K, group_size, bits,
                                _stream()), "dequantize")
    return out


def quantized_matmul(x, w, scales, biases, transpose: bool = True, group_size: int = 64, bits: int = 4):
    """mx.quantized_matmul (MLX/mlx/ops.cpp:3984-4021; validation :74-137), transpose=True only."""
    w = _as_words(w)
    if scales.shape != biases.shape:
        raise ValueError("[quantized_matmul] Scales and biases should have the same shape. Received scales with "
                         f"shape {tuple(scales.shape)} and biases with {tuple(biases.shape)}")
    if w.dim() < 2 or w.shape[:-1] != scales.shape[:-1]:
        raise ValueError("[quantized_matmul] Weight, scales and biases should have the same batch shape.")
    if w.shape[-1] * 32 // bits != scales.shape[-1] * group_size:
        raise ValueError("[quantized_matmul] The shapes of the weight and scales are incompatible based on bits and "
                         f"group_size. w.shape() == {tuple(w.shape)} and scales.shape() == {tuple(scales.shape)} "
                         f"with group_size={group_size} and bits={bits}")
    if not transpose:
        raise ValueError("[quantized_matmul] transpose=False is not on the QuantizedLinear path and is not built here")
    N, K = w.shape[-2], w.shape[-1] * 32 // bits
    if x.shape[-1] != K:
        raise ValueError(f"[quantized_matmul] Last dimension of first input with shape {tuple(x.shape)} does not "
                         f"match the expanded quantized matrix ({K}, {N}) computed from shape {tuple(w.shape)} with "
                         f"group_size={group_size}, bits={bits} and transpose=true")
    if not x.dtype.is_floating_point:
        raise ValueError("[quantized_matmul] Only real floating types are supported but x.dtype() == " f"{x.dtype}")
    _check_gs_bits("quantized_matmul", group_size, bits)
    if w.dim() != 2:
        raise ValueError("[quantized_matmul] batched weights are not built here")
    if x.dtype != _BF16 or scales.dtype != _BF16:
        raise ValueError("[quantized_matmul] only bfloat16 activations/scales/biases are built here")
    x2 = x.reshape(-1, K).contiguous()
    w, scales, biases = w.contiguous(), scales.contiguous(), biases.contiguous()
    M = x2.shape[0]
    y = torch.empty((M, N), dtype=_BF16, device=x.device)
    L = _lib.load()
    if group_size == 64 and bits in (4, 8) and qmt_scratch_bytes(M, N, K, bits, 0):
        seg = (QmvSeg * 1)()
        seg[0].wq, seg[0].scales, seg[0].biases, seg[0].N = w.data_ptr(), scales.data_ptr(), biases.data_ptr(), N
        if _qmt(y, x2, seg, 1, M, K, N, bits, None, 0.0, EPI_STORE, None, 0):
            return y.reshape(x.shape[:-1] + (N,))
    nb = _qmv_workspace_bytes(min(M, 32) if M else 1, N, K, bits, 0) if bits in (4, 8) and group_size == 64 else 0
    ws = qmv_workspace(nb, x.device)
    fn = L.pie_qmv if M <= 32 else L.pie_qmm
    _lib.check(fn(_p(y), _p(x2), _p(w), _p(scales), _p(biases), M, N, K, group_size, bits, _p(ws), ws.numel(),
                  _stream()), "quantized_matmul")
    return y.reshape(x.shape[:-1] + (N,))


def _segments(linears):
    """Segments of a launch, and the tensors they point into: held by the caller until the launch is queued, since another thread may put other
    tensors in a layer's place meanwhile."""
    held = [(lin.weight, lin.scales, lin.biases) for lin in linears]
    segs = (QmvSeg * len(held))()
    for seg, (w, s, b) in zip(segs, held):
        seg.wq, seg.scales, seg.biases, seg.N = w.data_ptr(), s.data_ptr(), b.data_ptr(), w.shape[0]
    return segs, held


def qmv_fused(x, linears, rows: int, K: int, N: int, bits: int, norm_weight, eps: float, residual, swiglu: bool):
    """pie_qmt or pie_qmv_fused on operands nn.fused_rows has checked.  N: output columns.  None: more than 32 rows that pie_qmt does not serve."""
    L = _lib.load()
    segs, held = _segments(linears)
    out = torch.empty(x.shape[:-1] + (N,), dtype=_BF16, device=x.device)
    epilogue = EPI_SILUMUL if swiglu else EPI_STORE if residual is None else EPI_RESADD
    if _qmt(out, x, segs, len(linears), rows, K, N, bits, norm_weight, float(eps), epilogue, residual, int(swiglu)):
        return out
    if rows > 32:
        return None
    ws = qmv_workspace(_qmv_workspace_bytes(rows, N, K, bits, int(swiglu)), x.device)
    _lib.check(L.pie_qmv_fused(_p(out), N, _p(x), K, rows, K, segs, len(linears), 64, bits, _p(norm_weight), float(eps), epilogue,
                               _p(residual), 0, _p(ws), ws.numel(), 2, _stream()), "qmv_fused")
    return out


def attention_workspace(units: int, nbytes: int, device) -> torch.Tensor:
    """Counters and partial sums of a decode step's attention over ``units`` (rows x query heads).  Keyed by the size of the counter region: the counters must
    be zero at a launch, and a buffer that served another (rows, heads) geometry holds that call's partial sums where this call's counters lie."""
    return workspaces.get(("attn", (units * 4 + 255) // 256), nbytes, device)


class _NoHost:
    """Where csrc/pie_host.cpp's module was not built, or for another torch or interpreter: None to every call."""
    mlp_rows = attend_rows = staticmethod(lambda *args: None)


@functools.cache
def native_fused_rows():
    """csrc/pie_host.cpp's form of nn.fused_rows, which takes the common calls and answers None to the others; where it was not built, or for another torch or
    interpreter, or for another of these libraries, so that it does not load or bind: None to every call."""
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_pie_host.so")
    if not os.path.exists(path):
        return lambda *args: None
    L = _lib.load()
    try:
        spec = importlib.util.spec_from_file_location("_pie_host", path)
        host = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(host)
        host.bind({name: C.cast(getattr(L, name), C.c_void_p).value for name in host.functions})
        host.fused_rows, host.mlp_rows, host.attend_rows
    except (ImportError, OSError, AttributeError, KeyError, TypeError) as e:   # (one of an earlier build has other functions, or another bind)
        warnings.warn(f"{path} does not load ({e}): build it again with make -C {_lib.CSRC}.  Calls of few rows take the Python form meanwhile.")
        return lambda *args: None
    return host.fused_rows


def native_host():
    """The module native_fused_rows() is of: several launches of few rows (mlp_rows, attend_rows), with the same None."""
    return getattr(native_fused_rows(), "__self__", _NoHost)


@functools.lru_cache(maxsize=4096)
def qmm_swiglu_pays(rows: int, N: int, K: int, bits: int) -> bool:
    return bool(_lib.load().pie_qmm_swiglu_pays(rows, N, K, 64, bits))


def qmm_swiglu(x, gate, up, rows: int, K: int):
    """pie_qmm_swiglu on operands nn.fused_swiglu has checked; None where the library leaves the shape to the separate calls."""
    segs, held = _segments((gate, up))
    out = torch.empty(x.shape[:-1] + (segs[0].N,), dtype=_BF16, device=x.device)
    status = _lib.load().pie_qmm_swiglu(_p(out), _p(x), segs, rows, K, 64, gate.bits, _stream())
    if status == _lib.EUNSUPPORTED:
        return None
    _lib.check(status, "qmm_swiglu")
    return out


def qmm_rows(x, linears, rows: int, K: int, N: int, residual):
    """pie_qmm_rows on operands nn.fused_prompt has checked; None where the library leaves them to the separate calls."""
    segs, held = _segments(linears)
    out = torch.empty(x.shape[:-1] + (N,), dtype=_BF16, device=x.device)
    status = _lib.load().pie_qmm_rows(_p(out), N, _p(x), segs, len(linears), _p(residual), rows, K, 64, linears[0].bits, _stream())
    if status == _lib.EUNSUPPORTED:
        return None
    _lib.check(status, "qmm_rows")
    return out


def rms_norm(x, weight, eps: float):
    """mx.fast.rms_norm (MLX/mlx/fast.cpp:56-123): bf16(bf16(x * rsqrt(mean(x^2) + eps)) * weight)."""
    if x.dim() < 1:
        raise ValueError("[rms_norm] Input must have at least 1 dimension but got input with 0 dimensions.")
    if weight is not None:
        if weight.dim() != 1:
            raise ValueError(f"[rms_norm] weight must have 1 dimension but has {weight.dim()} dimensions.")
        if weight.shape[0] != x.shape[-1]:
            raise ValueError("[rms_norm] weight must have the same size as the last dimension of x but has "
                             f"{weight.shape[0]} elements.")
        if weight.dtype != _BF16:
            raise ValueError("[rms_norm] only bfloat16 is built here")
        weight = weight.contiguous()
    if x.dtype != _BF16:
        raise ValueError("[rms_norm] only bfloat16 is built here")
    x = x.contiguous()
    out = torch.empty_like(x)
    dims = x.shape[-1]
    L = _lib.load()
    _lib.check(L.pie_rms_norm(_p(out), _p(x), _p(weight), x.numel() // dims if dims else 0, dims, float(eps),
                              _stream()), "rms_norm")
    return out


def rope(x, dims: int, *, traditional: bool = False, base: float | None = None, scale: float = 1.0,
         offset: int = 0, freqs: torch.Tensor | None = None):
    """mx.fast.rope (MLX/mlx/fast.cpp:353-511).  x [..., L, D]; all leading dims are flattened."""
    if x.dim() < 3:
        raise ValueError(f"[rope] Input must have at least 3 dimensions but got input with {x.dim()} dimensions.")
    if (base is None) == (freqs is None):
        raise ValueError("[rope] Only one of base or freqs can have a value.")
    if freqs is not None:
        if freqs.dim() != 1:
            raise ValueError(f"[rope] freqs must be one dimensional but has {freqs.dim()} dimensions.")
        if freqs.shape[0] != dims // 2:
            raise ValueError(f"[rope] freqs must have the same size as dims / 2 = {dims // 2} but has size "
                             f"{freqs.shape[0]}.")
        freqs = freqs.to(torch.float32).contiguous()
    if x.dtype != _BF16:
        raise ValueError("[rope] only bfloat16 is built here")
    Lq, D = x.shape[-2], x.shape[-1]
    L = _lib.load()
    if freqs is not None and not traditional and dims == D and D in (64, 128) and scale == 1.0 and x.dim() == 4 and _heads_ok(x) \
            and not (x.numel() <= 1024 * D and x.is_contiguous()):
        # the Llama case: every feature rotated, halves paired; heads may lie as the projection wrote them.  (Few rows that need no copy
        # are sooner done by the kernel with a thread per pair: 32 heads of 128, one token, 2.1 us for 2.9; the same bits.)
        B, H = x.shape[0], x.shape[1]
        out = torch.empty((B, H, Lq, D), dtype=_BF16, device=x.device)
        _lib.check(L.pie_rope_heads(_p(out), _p(x), B, H, Lq, D, x.stride(0), x.stride(1), x.stride(2), int(offset), _p(freqs),
                                    _stream()), "rope")
        return out
    x = x.contiguous()
    out = torch.empty_like(x)
    _lib.check(L.pie_rope(_p(out), _p(x), x.numel() // (Lq * D), Lq, D, dims, int(traditional),
                          0.0 if base is None else float(base), float(scale), int(offset), _p(freqs), _stream()),
               "rope")
    return out


def _heads_ok(x) -> bool:
    """[B, H, L, D] whose rows a kernel can read 16 bytes at a time wherever they lie."""
    return x.stride(3) == 1 and (x.stride(0) | x.stride(1) | x.stride(2)) % 8 == 0 and x.data_ptr() % 16 == 0 and x.shape[0] <= 65535


def kv_write(kbuf, vbuf, lay: "KvLayout", keys, values, offset: int):
    """keys, values [B, Hkv, L, D] -> cache rows offset .. offset + L - 1, from wherever their rows lie."""
    B, H, Lq, D = keys.shape
    if keys.stride(3) != 1:
        keys = keys.contiguous()
    if values.stride(3) != 1:
        values = values.contiguous()
    _lib.check(_lib.load().pie_kv_write_strided(_p(kbuf), _p(vbuf), C.byref(lay), _p(keys), keys.stride(0), keys.stride(1),
                                                keys.stride(2), _p(values), values.stride(0), values.stride(1), values.stride(2),
                                                B, H, Lq, D, offset, _stream()), "update_and_fetch")


def rope_kv_rows(queries, keys, values, freqs, offset: int, write):
    """Rotation of queries and keys [B, heads, L, D] at positions offset .. and the cache write of keys and values in one launch: the bits of rope of the
    two and kv_write / kvq_write.  ``write``: (kbuf, vbuf, KvLayout), or a KvqCache.  Returns the rotated queries, contiguous; None where the separate calls
    are to be made (which also report what is wrong)."""
    B, Hq, Lq, D = queries.shape
    Hkv = keys.shape[1]
    if D not in (64, 128) or keys.shape != (B, Hkv, Lq, D) or values.shape != keys.shape or freqs.dtype != torch.float32 or freqs.shape != (D // 2,) \
            or not freqs.is_contiguous() or not 0 < B <= 65535 or Hq + 2 * Hkv > 65535 or Lq == 0 \
            or any(t.dtype != _BF16 or not t.is_cuda or t.stride(3) != 1 for t in (queries, keys, values)):
        return None
    out = torch.empty((B, Hq, Lq, D), dtype=_BF16, device=queries.device)
    rows = [HeadRows(t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)) for t in (queries, keys, values)]
    L = _lib.load()
    if isinstance(write, KvqCache):
        status = L.pie_rope_kvq_rows(_p(out), C.byref(write), *map(C.byref, rows), None, _p(freqs), B, Hq, Hkv, Lq, D, int(offset), _stream())
        if status == _lib.EUNSUPPORTED:
            return None
    else:
        kbuf, vbuf, lay = write
        status = L.pie_rope_kv_rows(_p(out), _p(kbuf), _p(vbuf), C.byref(lay), *map(C.byref, rows), None, _p(freqs), B, Hq, Hkv, Lq, D, int(offset),
                                    _stream())
    _lib.check(status, "update_and_fetch")
    return out


class CausalMask:
    """What create_attention_mask returns for L > 1 (PIE/models/base.py:37-53): the additive -1e9 causal mask
    [L, offset + L], kept symbolic because the attention kernel builds it from (offset, L)."""

    def __init__(self, L: int, offset: int):
        self.L, self.offset = L, offset
        self.shape = (L, offset + L)


def kv_layout(k: torch.Tensor, page_table=None, page_size: int = 0) -> KvLayout:
    """Strides (elements) of a [B, Hkv, T, D] view of a cache buffer, or of a page pool [pages, page, Hkv, D]."""
    lay = KvLayout()
    if page_table is None:
        if k.stride(3) != 1:
            raise ValueError("[scaled_dot_product_attention] keys/values must be contiguous in the feature dimension")
        lay.batch_stride, lay.head_stride, lay.tok_stride = k.stride(0), k.stride(1), k.stride(2)
        lay.page_table, lay.pt_stride, lay.page_size = None, 0, 0
    else:
        lay.batch_stride, lay.head_stride, lay.tok_stride = 0, k.stride(2), k.stride(1)
        lay.page_table, lay.pt_stride, lay.page_size = page_table.data_ptr(), page_table.stride(0), page_size
    return lay


def decode_attention(q, kbuf, vbuf, lay: KvLayout, positions, scale: float, nsplit: int = 0, max_context: int = 0):
    """Decode-step attention on explicit cache geometry.  q [B, Hq, D]; positions int32 [B] (context = pos + 1)."""
    B, Hq, D = q.shape
    Hkv = kbuf.shape[1] if lay.page_table is None else kbuf.shape[2]
    L = _lib.load()
    if nsplit <= 0:
        nsplit = L.pie_decode_attn_pick_splits_for(B, Hq, Hkv, D, max_context if max_context > 0 else 1)
    nb = L.pie_decode_attn_workspace_bytes(B, Hq, D, nsplit)
    ws = attention_workspace(B * Hq, nb, q.device)
    out = torch.empty((B, Hq * D), dtype=_BF16, device=q.device)
    _lib.check(L.pie_decode_attn(_p(out), _p(q), _p(kbuf), _p(vbuf), C.byref(lay), _p(positions), B, Hq, Hkv, D,
                                 float(scale), nsplit, _p(ws), ws.numel(), _stream()), "scaled_dot_product_attention")
    return out


def scaled_dot_product_attention(q, k, v, *, scale: float, mask=None):
    """mx.fast.scaled_dot_product_attention (MLX/mlx/fast.cpp:566-783) for the two shapes the Llama path uses:
    L == 1 with mask None (decode) and L > 1 with the causal mask of create_attention_mask (prefill)."""
    for t in (q, k, v):
        if t.dim() != 4:
            raise ValueError(f"[scaled_dot_product_attention] input with shape {tuple(t.shape)} expected to be rank 4")
    B, Hq, Lq, D = q.shape
    if k.shape[0] != B or v.shape[0] != B:
        raise ValueError("[scaled_dot_product_attention] mismatching batch dimension for input")
    if k.shape[-1] != D:
        raise ValueError("[scaled_dot_product_attention] query, keys expected to have matching last dimension")
    Hkv, T = k.shape[1], k.shape[2]
    if v.shape[1] != Hkv:
        raise ValueError("[scaled_dot_product_attention] keys, values expected to have matching n_kv_heads")
    if Hq % Hkv != 0:
        raise ValueError("[scaled_dot_product_attention] n_heads must be a multiple of n_kv_heads")
    if q.dtype != _BF16 or k.dtype != _BF16 or v.dtype != _BF16:
        raise ValueError("[scaled_dot_product_attention] only bfloat16 is built here")
    # (the stride of a dimension of one element says nothing: a view of projected rows and a rotated copy of one differ there)
    if any(a != b and (n != 1 or m != 1) for n, m, a, b in zip(k.shape, v.shape, k.stride(), v.stride())):
        raise ValueError("[scaled_dot_product_attention] keys and values must share one layout")
    lay = kv_layout(k)
    L = _lib.load()
    if Lq == 1 and mask is None:
        pos = torch.full((B,), T - 1, dtype=torch.int32, device=q.device)
        out = decode_attention(q.reshape(B, Hq, D).contiguous(), k, v, lay, pos, scale, max_context=T)
        return out.view(B, Hq, 1, D)
    if isinstance(mask, str) and mask == "causal":
        mask = CausalMask(Lq, T - Lq)
    if not isinstance(mask, CausalMask):
        raise ValueError("[scaled_dot_product_attention] only mask=None (L == 1), 'causal' or the CausalMask of "
                         "create_attention_mask are built here")
    if mask.offset + mask.L != T or mask.L != Lq:
        raise ValueError("[scaled_dot_product_attention] mask shape does not match the keys")
    out = torch.empty((B, Lq, Hq * D), dtype=_BF16, device=q.device)
    _lib.check(L.pie_prefill_attn(_p(out), _p(q.contiguous()), _p(k), _p(v), C.byref(lay), B, Hq, Hkv, Lq, D,
                                  mask.offset, float(scale), _stream()), "scaled_dot_product_attention")
    return out.view(B, Lq, Hq, D).permute(0, 2, 1, 3)


def prefill_attention(q, kbuf, vbuf, lay: KvLayout, offset: int, scale: float):
    """Causal attention of L > 1 new tokens over a cache that already holds them (T = offset + L) on explicit cache
    geometry, contiguous or paged: chunked prefill / prefix reuse.  q [B, Hq, L, D] -> [B, Hq, L, D]."""
    B, Hq, Lq, D = q.shape
    Hkv = kbuf.shape[1] if lay.page_table is None else kbuf.shape[2]
    out = torch.empty((B, Lq, Hq * D), dtype=_BF16, device=q.device)
    _lib.check(_lib.load().pie_prefill_attn(_p(out), _p(q.contiguous()), _p(kbuf), _p(vbuf), C.byref(lay), B, Hq, Hkv, Lq, D,
                                            int(offset), float(scale), _stream()), "scaled_dot_product_attention")
    return out.view(B, Lq, Hq, D).permute(0, 2, 1, 3)


def kvq_desc(keys, values, page_table=None, page_size: int = 0, group_size: int = 64, bits: int = 8) -> KvqCache:
    """pie_kvq_cache over the (quants, scales, biases) triples of a quantised KV cache: contiguous
    [B, Hkv, cap, D/4 | D/64] (QuantizedKVCache's own arrays) or pools [pages, Hkv, page_size, .] + a page table."""
    d = KvqCache()
    for name, t in zip(("k_quant", "k_scales", "k_biases", "v_quant", "v_scales", "v_biases"), (*keys, *values)):
        if not t.is_contiguous():
            raise ValueError("quantised KV cache buffers must be contiguous")
        setattr(d, name, t.data_ptr())
    d.capacity = keys[0].shape[2]
    if page_table is None:
        d.page_table, d.pt_stride, d.page_size = None, 0, 0
    else:
        d.page_table, d.pt_stride, d.page_size = page_table.data_ptr(), page_table.stride(0), page_size
    d.group_size, d.bits = group_size, bits
    return d


def kvq_append(qkv, desc: KvqCache, positions, freqs, Hq: int, Hkv: int, D: int, q_out=None):
    """Decode step: rotate q and k of the fused projection output [B, (Hq + 2 Hkv) D] at positions[b], quantise k and v
    into the cache (QuantizedKVCache.update_and_fetch, PIE/cache/kv_cache/quantized.py:92-106).  Returns q [B, Hq, D]."""
    B = qkv.shape[0]
    if q_out is None:
        q_out = torch.empty((B, Hq, D), dtype=_BF16, device=qkv.device)
    _lib.check(_lib.load().pie_kvq_append(_p(q_out), _p(qkv), C.byref(desc), _p(positions), _p(freqs), B, Hq, Hkv, D,
                                          _stream()), "kvq_append")
    return q_out


def kvq_write(desc: KvqCache, keys, values, offset: int):
    """Quantise k, v [B, Hkv, L, D] into cache rows offset .. offset + L - 1."""
    B, Hkv, L, D = keys.shape
    kc, vc = keys.contiguous(), values.contiguous()
    _lib.check(_lib.load().pie_kvq_write(C.byref(desc), _p(kc), _p(vc), B, Hkv, L, D, offset, _stream()), "kvq_write")


def decode_attention_q8(q, desc: KvqCache, positions, scale: float, Hkv: int, nsplit: int = 0, max_context: int = 0,
                        out=None):
    """quantized_scaled_dot_product_attention for one query token (PIE/models/base.py:56-89) over a quantised cache.
    q [B, Hq, D]; positions int32 [B] (context = pos + 1) -> [B, Hq * D]."""
    B, Hq, D = q.shape
    L = _lib.load()
    if nsplit <= 0:
        nsplit = L.pie_decode_attn_q8_pick_splits(B, Hq, Hkv, max_context if max_context > 0 else 1)
    nb = L.pie_decode_attn_workspace_bytes(B, Hq, D, nsplit)
    ws = attention_workspace(B * Hq, nb, q.device)
    if out is None:
        out = torch.empty((B, Hq * D), dtype=_BF16, device=q.device)
    qc = q.contiguous()
    _lib.check(L.pie_decode_attn_q8(_p(out), _p(qc), C.byref(desc), _p(positions), B, Hq, Hkv, D, float(scale), nsplit,
                                    _p(ws), ws.numel(), _stream()), "decode_attn_q8")
    return out


def silu_mul(gate, up):
    """nn.silu(gate) * up with a bf16 rounding at each MLX op boundary (language.py:126-127)."""
    gate, up = gate.contiguous(), up.contiguous()
    out = torch.empty_like(gate)
    _lib.check(_lib.load().pie_silu_mul(_p(out), _p(gate), _p(up), gate.numel(), _stream()), "silu_mul")
    return out


def add(a, b):
    a, b = a.contiguous(), b.contiguous()
    out = torch.empty_like(a)
    _lib.check(_lib.load().pie_add(_p(out), _p(a), _p(b), a.numel(), _stream()), "add")
    return out


def argmax(logits, positions_to_advance=None, seq_out=None, out=None):
    """Greedy sampler (temp == 0): first arg-max of each row of bf16 logits [rows, vocab] -> int32 [rows]."""
    logits = logits.contiguous()
    rows, vocab = logits.shape
    if out is None:
        out = torch.empty((rows,), dtype=torch.int32, device=logits.device)
    _lib.check(_lib.load().pie_argmax(_p(out), _p(logits), rows, vocab, _p(positions_to_advance), _p(seq_out),
                                      0 if seq_out is None else seq_out.shape[1], _stream()), "argmax")
    return out


def new_rng_state(seed: int, device="cuda") -> torch.Tensor:
    """Device-resident Philox state of pie_sample: [seed, draw counter, scratch, scratch] (int64)."""
    return torch.tensor([int(seed) & 0x7FFFFFFFFFFFFFFF, 0, 0, 0], dtype=torch.int64, device=device)


def sample(logits, temp: float, top_p: float = 0.0, min_p: float = 0.0, min_tokens_to_keep: int = 1, top_k: int = -1,
           rng_state=None, uniforms=None, return_logprobs: bool = False, positions_to_advance=None, seq_out=None,
           out=None, logprobs_out=None):
    """The temperature branches of make_sampler (PIE/samplers/__init__.py:11-45) on bf16 logits [rows, vocab], in one
    launch together with logprobs = f32(logits) - logsumexp (inference_engine.py:268-269).  Returns tokens (int32 [rows])
    or (tokens, logprobs f32 [rows, vocab])."""
    if temp <= 0:
        raise ValueError("[sample] temp must be > 0 (temp == 0 is argmax)")
    if not (0 <= min_p <= 1.0):
        raise ValueError(f"`min_p` has to be a float in the [0, 1] interval, but is {min_p}")          # min_p.py:33-36
    if not isinstance(min_tokens_to_keep, int) or min_tokens_to_keep < 1:
        raise ValueError(f"`min_tokens_to_keep` has to be a positive integer, but is {min_tokens_to_keep}")  # :37-40
    logits = logits.contiguous()
    rows, vocab = logits.shape
    use_top_k = not (0 < top_p < 1.0) and min_p == 0.0 and top_k > 0
    if use_top_k and not (isinstance(top_k, int) and 0 < top_k < vocab):
        raise ValueError(f"`top_k` has to be an integer in the (0, {vocab}] interval, but is {top_k}.")  # top_k.py:23-27
    if logits.dtype != _BF16:
        raise ValueError("[sample] only bfloat16 logits are built here")
    if rng_state is None and uniforms is None:
        raise ValueError("[sample] needs rng_state (ops.new_rng_state) or uniforms")
    if out is None:
        out = torch.empty((rows,), dtype=torch.int32, device=logits.device)
    if return_logprobs and logprobs_out is None:
        logprobs_out = torch.empty((rows, vocab), dtype=torch.float32, device=logits.device)
    if uniforms is not None:
        uniforms = uniforms.to(torch.float32).contiguous()
    _lib.check(_lib.load().pie_sample(_p(out), _p(logits), rows, vocab, vocab, float(temp), float(top_p), float(min_p),
                                      int(min_tokens_to_keep), int(top_k), _p(rng_state), _p(uniforms), _p(logprobs_out),
                                      _p(positions_to_advance), _p(seq_out), 0 if seq_out is None else seq_out.shape[1],
                                      _stream()), "sample")
    return (out, logprobs_out) if return_logprobs else out


_VOID = ("a bounded wait inside a tensor-core pipeline expired: results since the last check that passed are void "
         "(and every check fails until {}_pipeline_error_clear())")


class PipelineWatch:
    """Whether a kernel gave up a wait, without a wait for it: post() behind a step's launches queues a copy of the library's word
    on the current stream, check() raises once a copy that said so has landed -- where the host has waited for the step anyway
    (its tokens are there), and before the next step."""

    _landings: dict = {}   # (library, device) -> the words: they say the same to every engine, and stay for copies still on their way

    def __init__(self, lib, prefix: str, page_locked: bool = True):
        self._words_fn, self._error_fn, self._prefix = getattr(lib, prefix + "_pipeline_words"), getattr(lib, prefix + "_pipeline_error"), prefix
        if page_locked:
            key = (prefix, torch.cuda.current_device())
            if key not in self._landings:
                self._landings[key] = torch.zeros(2, dtype=torch.int32, pin_memory=True)
            self.words = self._landings[key]
        else:
            self.words = torch.zeros(2, dtype=torch.int32)
        self._seen, self._at = self.words.numpy(), self.words.data_ptr()

    def post(self) -> None:
        if self._words_fn(self._at, _stream()):
            raise RuntimeError("[pipeline_words] CUDA error")

    def check(self) -> None:
        if self._seen[0] or self._seen[1]:
            if self._error_fn():         # still set (waits for the device): every engine is to hear of it, so the words stay
                raise RuntimeError(_VOID.format(self._prefix))
            self._seen[:] = 0            # cleared since


def check_pipeline() -> None:
    """The same for calls outside an engine (a layer, a model, attention): waits for the device."""
    if _lib.load().pie_pipeline_error():
        raise RuntimeError(_VOID.format("pie"))


def launch_count() -> int:
    return int(_lib.load().pie_launch_count())
