"""Activations behind the dense matmul, applied four values at a time: edges of a tile's rows and columns, with and without a bias, rows that are not aligned."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act", ["softcap", "tanh", "xielu", "gelu"])
@pytest.mark.parametrize("M,N,ld", [(64, 224, 224), (300, 258, 260), (300, 259, 259), (257, 33, 36), (1300, 2305, 2305)])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("bf16", [False, True])
def test_activations(act, M, N, ld, bias, bf16):
    """Against float64 of the same product and sums.  The sums differ by 2^-24 sum |x w| at most times a few, an activation's slope is at most 2 here, the functions
    are within a few units of 2^-24, and a bf16 result is rounded once."""
    from proxy_inference_engine_b200 import _lib
    L, K = _lib.load_hybrid(build_if_missing=True), 256
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = (torch.randn((n, K), generator=g, device="cuda").bfloat16() for n in (M, N))
    w = (w * (2 / K ** 0.5)).bfloat16()
    b = torch.randn(N, generator=g, device="cuda") if bias else None
    out = torch.full((M, ld), 7.0, device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)
    p = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    kind, a0, a1 = {"softcap": (_lib.EPI_SOFTCAP, 3.0, 0.0), "tanh": (_lib.EPI_TANH, 0.0, 0.0), "xielu": (_lib.EPI_XIELU, 0.8, 0.3), "gelu": (_lib.EPI_GELU, 0.0, 0.0)}[act]
    if act == "softcap":
        assert L.pieh_linear(p(out), 0 if bf16 else 1, ld, p(x), 0, K, p(w), 0, p(b), M, N, K, kind, a0, None, None, 0, None) == 0
    else:
        assert L.pieh_linear_act(p(out), 0 if bf16 else 1, ld, p(x), 0, K, p(w), 0, p(b), M, N, K, kind, a0, a1, None) == 0
    z = x.double() @ w.double().T + (b.double() if bias else 0)
    mass = x.double().abs() @ w.double().abs().T + z.abs()
    want = {"softcap": lambda: a0 * torch.tanh(z / a0), "tanh": lambda: torch.tanh(z),
            "xielu": lambda: torch.where(z > 0, a0 * z * z, a1 * (torch.expm1(z) - z)) + z / 2,
            "gelu": lambda: z / 2 * (1 + torch.tanh((2 / torch.pi) ** 0.5 * (z + 0.044715 * z ** 3)))}[act]()
    slope = 2 * a0 * z.abs() + 1 if act == "xielu" else 2
    bound = slope * 2 ** -20 * mass + (2 ** -8 if bf16 else 2 ** -20) * want.abs()
    assert ((out[:, :N].double() - want).abs() <= bound).all()
    assert (out[:, N:] == 7).all()
