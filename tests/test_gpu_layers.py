"""The Llama layers' calls on the GPU, in the forms that whole-model tests do not reach."""
import pytest
import torch

from parity_util import tiny_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("B,L", [(1, 1), (3, 1), (1, 40), (3, 40)])   # fused rows, then separate calls
def test_a_model_without_a_cache_is_the_one_with_an_empty_cache(head_dim, B, L):
    from proxy_inference_engine_b200.checkpoint import build_model, random_weights
    args = tiny_args(bits=4, head_dim=head_dim)
    model = build_model(args, random_weights(args, seed=0, device="cuda"))
    ids = torch.randint(0, args.vocab_size, (B, L), generator=torch.Generator().manual_seed(L)).cuda().to(torch.int32)
    assert torch.equal(model(ids), model(ids, cache=model.make_cache()))


def test_the_engines_bring_the_pipelines_word_to_the_host():
    """Whatever the words hold, a prompt overwrites them with the library's own (0: no wait expired) by the time its tokens are read, and
    words that say otherwise are checked with the library."""
    from proxy_inference_engine_b200.checkpoint import build_model, random_weights
    from proxy_inference_engine_b200.decode import DecodeEngine
    args = tiny_args(bits=4)
    eng = DecodeEngine(build_model(args, random_weights(args, seed=0, device="cuda")), batch=1, max_context=128)
    eng.watch.words.fill_(-1)
    eng.prefill(torch.arange(70))
    assert eng.generated().shape == (1, 1) and eng.watch.words.tolist() == [0, 0]
    eng.watch.words.fill_(-1)
    eng.step()
    assert eng.watch.words.tolist() == [0, 0]


def test_silu_of_every_gate():
    """All bf16 gates: the bits of sigmoid and product in full fp32, rounded to bf16 after each (subnormal sigmoids among them)."""
    from proxy_inference_engine_b200 import ops
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    sig = (1 / (1 + torch.exp(-g.float()))).to(torch.bfloat16)
    want = (g.float() * sig.float()).to(torch.bfloat16)
    got = ops.silu_mul(g.cuda(), torch.ones_like(g).cuda()).cpu()
    nan = want.isnan()
    assert torch.equal(nan, got.isnan()) and torch.equal(got[~nan].view(torch.int16), want[~nan].view(torch.int16))


def _linear(N, K, bits, g):
    from proxy_inference_engine_b200 import nn, ops
    lin = object.__new__(nn.QuantizedLinear)
    lin.group_size, lin.bits = 64, bits
    lin.weight, lin.scales, lin.biases = ops.quantize(torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16) / K ** 0.5, 64, bits)
    shifts = torch.arange(0, 32, bits, device="cuda", dtype=torch.int32)
    q = ((lin.weight[:, :, None] >> shifts) & (2 ** bits - 1)).reshape(N, K // 64, 64).double()
    lin.dense = (q * lin.scales.double()[:, :, None] + lin.biases.double()[:, :, None]).reshape(N, K)   # these kernels keep the exact codes
    lin.codes = (q * lin.scales.double()[:, :, None]).abs().sum((1, 2))
    return lin


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 32])          # either side of the kernels' row counts
@pytest.mark.parametrize("widths,K", [((48, 16, 7), 512),        # ragged tiles
                                      ((256, 128, 128), 512),    # whole ones: the 8-bit tensor-core kernel from nine rows on
                                      ((100, 100), 4096),        # K cut between warps and CTAs
                                      ((16384, 16384), 256)])    # from 17 rows on the batched tensor-core kernel
def test_fused_rows_against_the_separate_operators(bits, rows, widths, K):
    """One matrix, with or without a residual, is the separate calls bit for bit.  A norm in front, matrices side by side and SwiGLU
    sum in another order: those against float64."""
    from proxy_inference_engine_b200 import nn, ops
    g = torch.Generator(device="cuda").manual_seed(rows + K + bits + len(widths))
    lins = [_linear(N, K, bits, g) for N in widths]
    x = torch.randn((rows, K), generator=g, device="cuda").to(torch.bfloat16)
    res = torch.randn((rows, widths[0]), generator=g, device="cuda").to(torch.bfloat16)
    assert torch.equal(nn.fused_rows(x, lins[:1]), lins[0](x))
    assert torch.equal(nn.fused_rows(x, lins[:1], residual=res), ops.add(res, lins[0](x)))
    norm = nn.RMSNorm(K, eps=1e-5)
    norm.weight = (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).to(torch.bfloat16)
    xd = x.double()
    n = (xd * torch.rsqrt((xd ** 2).mean(-1, keepdim=True) + 1e-5)).to(torch.bfloat16).double() * norm.weight.double()
    n = n.to(torch.bfloat16).double()

    integer = bits == 8 and rows > 8 and K % 512 == 0 and all(N % 128 == 0 for N in widths)
    rounded = bits == 8 and rows > 16 and sum(widths) >= 16384      # the batched tensor-core kernel multiplies bf16(scale * code + bias)
    for lin in lins if rounded else ():
        lin.dense = lin.dense.to(torch.bfloat16).double()

    def product(v, lin, flips):
        """v W^T and how far an fp32 sum in any order may be from it; a normed value within 2^-22 of a rounding boundary may fall on
        the other side of it: 2^-13 of them, so hardly ever more than eight in a row, each by 2^-7 of itself."""
        w = lin.dense
        most = (v.abs()[:, :, None] * w.abs().t()[None]).amax(1) if w.numel() * rows < 2 ** 26 else v.abs().amax(-1, keepdim=True) * w.abs().amax(-1)
        # the integer tensor cores read a row as 15-bit fixed point, to half a step of 2^-14 of its largest value, and multiply scale * code by it
        fixed = 2 ** -15 * v.abs().amax(-1, keepdim=True) * lin.codes if integer else 0
        # (a weight it rounds in fp32 arithmetic may fall on the other side: 2^-7 of it, a few in a thousand, as in the tile kernels' test)
        return v @ w.t(), (v.abs() @ w.abs().t()) * (K * 2 ** -23 + (2 ** -15 if rounded else 0)) + (8 * 2 ** -7 * most if flips else 0) + fixed

    def within(got, want, slack):
        off = (got.double() - want).abs() - slack
        assert torch.isfinite(got).all() and off.max() <= 0, float(off.max())

    got, at = nn.fused_rows(x, lins, norm=norm), 0
    for lin, N in zip(lins, widths):
        y, slack = product(n, lin, True)
        within(got[:, at:at + N], y, slack + y.abs() * 2 ** -8)
        at += N
    if widths[0] == widths[1]:
        for v, kw in ((xd, {}), (n, {"norm": norm})):
            (a, da), (b, db) = (product(v, lin, bool(kw)) for lin in lins)
            da, db = da + a.abs() * 2 ** -8, db + b.abs() * 2 ** -8
            silu = a * torch.sigmoid(a)
            within(nn.fused_rows(x, lins, swiglu=True, **kw), silu * b,
                   1.1 * da * (b.abs() + db) + (silu.abs() + 1.1 * da) * db + 3.1 * 2 ** -8 * (silu * b).abs())


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("kv_bits", [None, 8])
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("B,L", [(1, 1), (8, 1), (9, 1), (32, 1), (33, 1), (2, 9)])
def test_a_block_of_few_rows_is_its_separate_operators(monkeypatch, bits, kv_bits, head_dim, B, L):
    """Attention, cache and feed-forward of a whole layer, two steps, with and without the fused calls.  Every result is rounded to bf16
    where the separate calls round, and what falls on the other side of a boundary is off by 2^-8 of itself."""
    from proxy_inference_engine_b200 import nn
    from proxy_inference_engine_b200.checkpoint import build_model, random_weights
    from proxy_inference_engine_b200.llama import create_attention_mask
    args = tiny_args(bits=bits, head_dim=head_dim, num_hidden_layers=1, hidden_size=512, num_attention_heads=512 // head_dim)
    model = build_model(args, random_weights(args, seed=0, device="cuda"))
    block, x = model.layers[0], torch.randn((2, B, L, 512), generator=torch.Generator(device="cuda").manual_seed(B + L), device="cuda").to(torch.bfloat16)
    fused, outs = nn.fused_rows, []
    calls = []
    for f in (lambda *a, **k: calls.append(1) or fused(*a, **k), lambda *a, **k: None):
        monkeypatch.setattr(nn, "fused_rows", f)
        cache = model.make_cache(kv_bits=kv_bits)
        outs.append(torch.stack([block(h, create_attention_mask(h, cache), cache[0]) for h in x]).double())
        assert cache[0].offset == 2 * L
    assert len(calls) == (8 if B * L <= 32 else 4)   # 33 rows: the layer asks once for its norm and projections and the feed-forward once
    assert (outs[0] - outs[1]).norm() <= 2 ** -8 * outs[1].norm()
