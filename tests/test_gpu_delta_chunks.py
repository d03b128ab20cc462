"""The gated delta rule 32 tokens at a time against the recurrence in float64, a token at a time, and against the kernel that takes them one by one."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _exact(q, k, v, beta, decay, S):
    """[n, H, .] in float64; S [H, dk, dv] -> (o, S)"""
    out = torch.empty_like(v)
    for t in range(len(v)):
        S = S * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hk,hkv->hv", k[t], S))
        S = S + torch.einsum("hk,hv->hkv", k[t], u)
        out[t] = torch.einsum("hk,hkv->hv", q[t], S)
    return out, S


def _run(seqs, H, G, dk, dv, ctx, seed, edit=None, keys="spread"):
    """seqs: rows of each sequence.  -> (chunks', one by one's, float64's) each (o, states), and the inputs"""
    from proxy_inference_engine_b200 import _lib
    from proxy_inference_engine_b200.ragged import BatchDetails
    L, n, T = _lib.load_hybrid(build_if_missing=True), len(seqs), sum(seqs)
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    base = 3 * rnd(1, G, dk) if keys == "alike" else 0          # nearly parallel keys: the triangle is far from the identity
    q, k, v = unit(rnd(T, G, dk) + base) / dk ** 0.5, unit(rnd(T, G, dk) + base), rnd(T, H, dv)
    beta = torch.sigmoid(rnd(T, H) + (2 if keys == "alike" else 0))
    decay = torch.exp(-torch.rand((T, H), generator=g, device="cuda") * torch.logspace(-3, 2, H, device="cuda"))     # from next to 1 to next to 0
    state = rnd(n, H, dk, dv)
    if edit:
        edit(q, k, v, beta, decay, state)
    b = BatchDetails.build([(str(i), [1] * m, ctx, list(range((ctx + m + 63) // 64)), i) for i, m in enumerate(seqs)])
    desc, keep = b.hybrid_descriptor()
    got = []
    for chunks in (True, False):
        st, o = state.clone(), torch.full((T, H, dv), float("nan"), device="cuda")
        d = _lib.HybDelta(H, G, dk, dv, 1, None, None, None, None, 1e-6, None, st.data_ptr())
        common = (_p(o), _p(q), _p(k), _p(v), _p(beta), _p(decay), C.byref(d), C.byref(desc))
        if chunks:
            nb = T * H * (2 * dk + dv + 2) * 4
            scratch = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")
            assert L.pieh_delta_scan_chunks(*common, _p(scratch), nb - 1, None) == 7      # PIE_EWORKSPACE
            assert L.pieh_delta_scan_chunks(*common, _p(scratch), nb, None) == 0
        else:
            assert L.pieh_delta_scan(*common, None) == 0
        torch.cuda.synchronize()
        got.append((o, st))
    rep, at, outs, sts = H // G, 0, [], []
    for i, m in enumerate(seqs):
        w = lambda x: x[at:at + m].double()
        o, s = _exact(w(q).repeat_interleave(rep, 1), w(k).repeat_interleave(rep, 1), w(v), w(beta), w(decay),
                      state[i].double() if ctx else torch.zeros_like(state[i]).double())
        outs.append(o)
        sts.append(s)
        at += m
    del keep
    return got[0], got[1], (torch.cat(outs), torch.stack(sts))


def _off(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("ctx", [0, 70])
@pytest.mark.parametrize("seqs", [[1], [2], [31], [32], [33], [64], [65], [96, 1, 130], [400]])     # edges of chunks and of tiles of two
@pytest.mark.parametrize("H,G,dk,dv", [(4, 4, 128, 128), (4, 2, 64, 20), (2, 1, 36, 4), (3, 3, 100, 48)])
def test_chunks_are_the_recurrence(H, G, dk, dv, seqs, ctx):
    """No further from float64 than a token at a time is, up to what the two orders of 32 + dk terms differ by: 2^-24 sqrt(32 + dk) is 8e-7."""
    mine, theirs, want = _run(seqs, H, G, dk, dv, ctx, sum(seqs) + dk)
    for a, b, w in zip(mine, theirs, want):
        assert _off(a, w) <= _off(b, w) + 8e-7


def test_keys_that_are_alike():
    """A of size one below the diagonal: solving the triangle must not lose what a token at a time keeps; 2e-7 is three roundings of 2^-24 on top."""
    mine, theirs, want = _run([700], 8, 8, 128, 128, 0, 5, keys="alike")
    for a, b, w in zip(mine, theirs, want):
        assert _off(a, w) <= 1.5 * _off(b, w) + 2e-7


@pytest.mark.parametrize("what", ["v", "k", "q", "beta", "decay", "state"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_what_is_no_number_spoils_what_comes_after_it_and_nothing_else(what, value):
    """In the middle of a chunk: the same places as a token at a time, and the others as they are without it."""
    at = {"q": 0, "k": 1, "v": 2, "beta": 3, "decay": 4, "state": 5}[what]

    def edit(*tensors):
        t = tensors[at]
        if what == "state":
            t[0, 1, 5, 3] = value
        elif what in ("beta", "decay"):
            t[45, 1] = value
        else:
            t[45, 1, 7] = value

    mine, theirs, _ = _run([100], 4, 4, 64, 32, 8, 7, edit=edit)
    clean = _run([100], 4, 4, 64, 32, 8, 7)[0]
    for a, b, c in zip(mine, theirs, clean):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
        hit = ~b.isfinite()
        assert torch.equal(a[hit].nan_to_num(0), b[hit].nan_to_num(0))
        fine = ~hit
        assert (a[fine] - b[fine]).abs().max() < 1e-4
    assert torch.equal(mine[0][:32], clean[0][:32]) or what == "state"


def test_the_rule_leaves_to_single_tokens_what_it_cannot_take():
    from proxy_inference_engine_b200 import _lib
    from proxy_inference_engine_b200.ragged import BatchDetails
    L = _lib.load_hybrid(build_if_missing=True)

    def scratch(rows, dk, dv):
        b = BatchDetails.build([(str(i), [1] * m, 0, list(range((m + 63) // 64)), i) for i, m in enumerate(rows)])
        desc, keep = b.hybrid_descriptor()
        return L.pieh_delta_scan_scratch(C.byref(_lib.HybDelta(4, 4, dk, dv, 1, None, None, None, None, 1e-6, None, None)), C.byref(desc))

    assert scratch([1200], 128, 128) == 1200 * 4 * (3 * 128 + 2) * 4
    for rows, dk, dv in (([1], 128, 128), ([1] * 300, 128, 128), ([1200], 129, 128), ([1200], 132, 128), ([1200], 128, 130), ([90000], 128, 128)):
        assert scratch(rows, dk, dv) == 0
