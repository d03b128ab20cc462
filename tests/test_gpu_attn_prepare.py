"""Rotation, norm and page writes of a step's rows: CTAs of eight warps for few rows, of four for many."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,d,dv,rot", [(1, 1, 64, 64, 64), (5, 1, 32, 128, 16), (16, 4, 64, 128, 64)])      # fewer units than warps, an odd number, many
@pytest.mark.parametrize("cache", ["bf16", "fp32"])
def test_rows_are_the_same_in_any_portions(H, G, d, dv, rot, cache):
    """700 rows at once (more than run together), and 592 and 108 of them: a unit is one warp's either way, so the bits are the same."""
    from proxy_inference_engine_b200 import _lib
    from proxy_inference_engine_b200.ragged import BatchDetails
    L, T = _lib.load_hybrid(build_if_missing=True), 700
    g = torch.Generator(device="cuda").manual_seed(H)
    proj = torch.randn((T, 2 * (H + G) * d + G * dv), generator=g, device="cuda")
    qn, kn = torch.rand(d, generator=g, device="cuda"), torch.rand(d, generator=g, device="cuda")
    freqs = torch.logspace(0, -4, rot // 2, dtype=torch.float64, device="cuda")
    pages, p = list(range((T + 63) // 64)), lambda t: C.c_void_p(t.data_ptr())
    got = []
    for portions in ([T], [592, T - 592]):
        kp, vp = (torch.zeros((len(pages), 64, G, w), dtype=torch.bfloat16 if cache == "bf16" else torch.float32, device="cuda") for w in (2 * d, dv))
        at = _lib.HybAttn(H, G, d, dv, rot, freqs.data_ptr(), qn.data_ptr(), kn.data_ptr(), 1e-6, 0.5, 0.0, 0, 0.4, 0.8, kp.data_ptr(), vp.data_ptr(),
                          0 if cache == "bf16" else 1)
        out, ctx = [], 0
        for n in portions:
            desc, keep = BatchDetails.build([("s", [0] * n, ctx, pages, 0)], device="cuda").hybrid_descriptor()
            q, part = torch.empty((n, H, 2, d), device="cuda"), proj[ctx:ctx + n]
            assert L.pieh_attn_prepare(p(q), p(part), part.stride(0), C.byref(at), C.byref(desc), None) == 0
            torch.cuda.synchronize()
            out.append(q)
            ctx += n
        got.append((torch.cat(out), kp, vp))
        del keep
    assert all(torch.equal(a, b) for a, b in zip(*got)) and got[0][0].isfinite().all()
