"""Host side of the Llama layers' calls: what reaches the library and what is refused, on CPU tensors with the library stubbed."""
import pytest
import torch

from proxy_inference_engine_b200 import ops


def _bf16(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16)


def test_one_key_may_be_a_view_and_a_copy(monkeypatch):
    """One token without a cache: rotated keys are a copy, values a view of the projection's rows.  They differ in the stride of a
    dimension of one element, which says nothing; any other difference is refused."""
    H, D = 2, 64
    monkeypatch.setattr(ops._lib, "load", lambda: None)
    monkeypatch.setattr(ops, "decode_attention", lambda q, *a, **k: torch.zeros(q.shape[0], q.shape[1] * q.shape[2]))
    view = lambda B, width: _bf16(B, 1, width)[..., :H * D].reshape(B, 1, H, D).transpose(1, 2)
    for B, width in ((1, H * D), (1, 3 * H * D), (3, H * D)):
        q, k, v = _bf16(B, H, 1, D), _bf16(B, H, 1, D), view(B, width)
        assert k.stride() != v.stride()
        assert ops.scaled_dot_product_attention(q, k, v, scale=1.0).shape == (B, H, 1, D)
    with pytest.raises(ValueError, match="one layout"):   # rows of another width: the batch stride counts
        ops.scaled_dot_product_attention(q, k, view(3, 3 * H * D), scale=1.0)
    with pytest.raises(ValueError, match="one layout"):
        ops.scaled_dot_product_attention(_bf16(1, H, 1, D), _bf16(1, H, 5, D), _bf16(1, 5, H, D).transpose(1, 2), scale=1.0)
