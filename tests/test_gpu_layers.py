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
