"""Decode attention in any number of splits: what the last CTA makes of their partial results."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(q, k, v, size, n):
    """float64: softmax over the first n[b] keys, and the sum of the probabilities times the size of what they multiply"""
    rep = q.shape[1] // k.shape[1]
    k, v, size = (t.double().repeat_interleave(rep, 1) for t in (k, v, size))
    s = torch.einsum("bhd,bhtd->bht", q.double(), k) * q.shape[-1] ** -0.5
    s = s.masked_fill(torch.arange(k.shape[2], device="cuda")[None, None] >= n[:, None, None], float("-inf"))
    p = s.softmax(-1)
    return torch.einsum("bht,bhtd->bhd", p, v), torch.einsum("bht,bhtd->bhd", p, size)


@pytest.mark.parametrize("nsplit", [2, 7, 8, 9, 31, 32, 33, 64, 100])      # trips of eight, lanes of a warp; more splits than there are keys
@pytest.mark.parametrize("kind,Hq,Hkv,D", [("bf16", 8, 2, 128), ("bf16", 6, 2, 64), ("bf16", 40, 2, 128), ("bf16", 17, 1, 64),
                                           ("q8", 8, 2, 128), ("q8", 5, 1, 128), ("q8", 24, 2, 128), ("q8", 6, 2, 64)])
def test_splits_add_up(kind, Hq, Hkv, D, nsplit):
    """Against float64 on the cache's own values.  A probability is rounded to bf16 (2^-8) or, times the scale of v = scale * quant + bias, to
    f16, the sums are fp32, and the result is rounded to bf16: |error| <= 2^-8 |o| + 2^-8 sum p |v|, for the other |scale * quant| + |bias| in the place of
    |v|.  Twice, as the counters have to be zero again; and the two are the same bits."""
    from proxy_inference_engine_b200 import ops
    from proxy_inference_engine_b200.cache import KVCache, QuantizedKVCache
    if kind == "bf16" and nsplit > 32 and Hq // Hkv <= 16:
        nsplit = 32
    g = torch.Generator(device="cuda").manual_seed(nsplit + D)
    T, pos = 700, torch.tensor([699, 0, 63, 330], dtype=torch.int32, device="cuda")
    q, k, v = (torch.randn((4, *s, D), generator=g, device="cuda").bfloat16() for s in ((Hq,), (Hkv, T), (Hkv, T)))
    if kind == "q8":
        cache = QuantizedKVCache(64, 8, T + 2)
        got = cache.update_and_fetch(k, v)
        parts = [(s.double().repeat_interleave(64, -1) * w.contiguous().view(torch.uint8).double(), b.double().repeat_interleave(64, -1)) for w, s, b in got]
        (k, v), size = (x + b for x, b in parts), parts[1][0].abs() + parts[1][1].abs()
        run = lambda: ops.decode_attention_q8(q, cache.desc(), pos, D ** -0.5, Hkv, nsplit=nsplit)
    else:
        cache = KVCache(T + 2)
        cache.update_and_fetch(k, v)
        size = v.abs()
        run = lambda: ops.decode_attention(q, cache.keys, cache.values, ops.kv_layout(cache.keys), pos, D ** -0.5, nsplit=nsplit)
    one, two = run(), run()
    o, mass = _exact(q, k, v, size, pos + 1)
    assert torch.equal(one, two)
    assert ((one.double().reshape(o.shape) - o).abs() <= 2 ** -8 * o.abs() + 2 ** -8 * mass).all()
