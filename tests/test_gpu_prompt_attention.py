"""Prompt attention where a CTA has several items of 256 rows to walk: every item's rows against float64, with last items of one query tile, of one row, and
pages whose last slots hold anything."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(q, k, v, offset, scale):
    B, Hq, L, D = q.shape
    rep = Hq // k.shape[1]
    seen = torch.arange(offset + L, device="cuda")[None] <= torch.arange(offset, offset + L, device="cuda")[:, None]
    out = torch.empty((B, Hq, L, D), dtype=torch.float64, device="cuda")
    for b in range(B):
        for h in range(Hq):
            s = (q[b, h].double() @ k[b, h // rep].double().t() * scale).masked_fill(~seen, -torch.inf)
            out[b, h] = torch.softmax(s, -1) @ v[b, h // rep].double()
    return out


# items: B x 32 heads x ceil(L / 256); 148 SMs
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,L,offset", [(5, 1, 2000),        # one row each, more than one a CTA, seventeen key tiles
                                        (3, 257, 0),         # a second item of one row
                                        (4, 384, 1000),      # a last item of one query tile, behind a prefix that is no whole tile
                                        (2, 1100, 77), (1, 2303, 0)])
@pytest.mark.parametrize("paged", [False, True])
def test_items_of_a_cta(D, B, L, offset, paged):
    from proxy_inference_engine_b200 import _lib, ops
    if L == 1:
        L = 2                                                # (one row is a decode step's)
    g = torch.Generator(device="cuda").manual_seed(B * L + D)
    T, Hq, Hkv = offset + L, 32, 4
    q, k, v = (s * torch.randn((B, H, n, D), generator=g, device="cuda") for s, H, n in ((1.5, Hq, L), (1.5, Hkv, T), (1.0, Hkv, T)))
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    scale = D ** -0.5
    if paged:
        pages = (T + 63) // 64
        table = torch.randperm(B * pages, generator=torch.Generator().manual_seed(L)).to(torch.int32).view(B, pages).cuda()
        pools = [torch.full((B * pages, 64, Hkv, D), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in "kv"]
        t = torch.arange(T, device="cuda")
        for pool, x in zip(pools, (k, v)):
            for b in range(B):
                pool[table[b, t // 64].long(), t % 64] = x[b].transpose(0, 1)
        got = ops.prefill_attention(q, *pools, ops.kv_layout(pools[0], table, 64), offset, scale)
    else:
        got = ops.scaled_dot_product_attention(q, k, v, scale=scale, mask=ops.CausalMask(L, offset))
    want = _exact(q, k, v, offset, scale)
    # probabilities and results in bf16 (2^-9 each of what they multiply or are), the sums in fp32
    assert torch.isfinite(got).all() and (got.double() - want).norm() <= 2 ** -8 * want.norm()
    assert (got.double() - want).abs().amax((2, 3)).max() <= 0.03
    assert _lib.load().pie_pipeline_error() == 0
