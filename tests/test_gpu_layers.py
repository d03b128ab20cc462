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
