"""The gated delta rule against the recurrence in float64 on keys that all but coincide, where an update undoes the one before it."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _unit(x):
    return x / x.norm(dim=-1, keepdim=True)


def _inputs(T, H, dk, dv, cos, decay, seed):
    """Keys (and queries) of cosine ``cos`` to one another, updates that replace 0.95 of what is stored, decays of exp(-u decay)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    uni = lambda *s: torch.rand(s, generator=g, device="cuda")
    base, off = _unit(rnd(1, H, dk)), (1 / cos - 1) ** 0.5
    q, k = (_unit(base + off * rnd(T, H, dk) / dk ** 0.5) for _ in "qk")
    return q / dk ** 0.5, k, rnd(T, H, dv), 0.94 + 0.02 * uni(T, H), torch.exp(-decay * uni(T, H))


def _scan(x, seqs):
    from proxy_inference_engine_b200 import _lib
    from proxy_inference_engine_b200.ragged import BatchDetails
    L = _lib.load_hybrid(build_if_missing=True)
    q, k, v, beta, decay = x
    (T, H, dk), dv = q.shape, v.shape[2]
    b = BatchDetails.build([(str(i), [1] * n, 0, list(range((n + 63) // 64)), i) for i, n in enumerate(seqs)])
    desc, keep = b.hybrid_descriptor()
    o, state = torch.full((T, H, dv), float("nan"), device="cuda"), torch.full((len(seqs), H, dk, dv), float("nan"), device="cuda")
    d = _lib.HybDelta(H, H, dk, dv, 1, None, None, None, None, 1e-6, None, state.data_ptr())
    assert L.pieh_delta_scan(_p(o), _p(q), _p(k), _p(v), _p(beta), _p(decay), C.byref(d), C.byref(desc), None) == 0
    torch.cuda.synchronize()
    del keep
    return o, state


def _exact(q, k, v, beta, decay):
    q, k, v, beta, decay = (t.double() for t in (q, k, v, beta, decay))
    S, o = torch.zeros((q.shape[1], q.shape[2], v.shape[2]), dtype=torch.float64, device="cuda"), torch.empty_like(v)
    for t in range(len(v)):
        S = S * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hk,hkv->hv", k[t], S))
        S = S + torch.einsum("hk,hv->hkv", k[t], u)
        o[t] = torch.einsum("hk,hkv->hv", q[t], S)
    return o, S


@pytest.mark.parametrize("cos", [0.9, 0.99, 0.999])
@pytest.mark.parametrize("T,dk,dv", [(300, 128, 128), (400, 64, 48)])
def test_keys_that_coincide(cos, T, dk, dv):
    """A read-out is a sum of dk products of fp32 whose largest cancel nothing, and what is stored wrongly of a token the next update takes back: an error of two
    roundings of 2^-24 (1.2e-7) in the outputs, where every 32 tokens solved for together are off by 1.8e-7 and more."""
    x = _inputs(T, 8, dk, dv, cos, 0.1, T)
    (o, S), (wo, wS) = _scan(x, [T]), _exact(*x)
    assert float((o.double() - wo).norm() / wo.norm()) <= 2 * 2 ** -24
    assert float((S[0].double() - wS).norm() / wS.norm()) <= 4 * 2 ** -24


def test_a_prompt_is_the_same_beside_others():
    """Bit for bit, beside a sequence that decodes one token and another prompt."""
    x = _inputs(300 + 1 + 40, 4, 128, 64, 0.9, 0.1, 3)
    o, S = _scan(x, [300, 1, 40])
    alone = _scan([t[:300].contiguous() for t in x], [300])
    assert torch.equal(o[:300], alone[0]) and torch.equal(S[:1], alone[1])
