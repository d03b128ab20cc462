"""How a DecodeEngine attends follows from its room, and stands for every position in it."""
import pytest

from parity_util import tiny_args

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from proxy_inference_engine_b200.checkpoint import build_model, random_weights
    from proxy_inference_engine_b200.decode import DecodeEngine
    models = {}

    def make(D, *a, **kw):
        if D not in models:
            args = tiny_args(head_dim=D, hidden_size=512, num_attention_heads=32, num_key_value_heads=8, num_hidden_layers=1)
            models[D] = build_model(args, random_weights(args, seed=0, device="cuda"))
        return DecodeEngine(models[D], *a, **kw)

    return make


@pytest.mark.parametrize("batch,room,one", [(1, 64, True), (1, 4096, True), (1, 4097, False), (4, 1024, True), (4, 1025, False), (32, 128, True), (32, 129, False)])
def test_one_launch_up_to_4096_keys(engine, batch, room, one):
    assert engine(128, batch, room).attn_fused == one


@pytest.mark.parametrize("D,kv_bits,batch,room,splits", [(128, 8, 1, 1023, 1), (128, 8, 1, 1024, 8), (64, 8, 8, 600, 1), (128, 8, 32, 2048, 1), (64, None, 32, 2048, 1),
                                                         (64, None, 16, 2048, 4), (128, None, 16, 2048, 2), (128, None, 1, 64, 1)])
def test_splits_only_where_they_pay_soon(engine, D, kv_bits, batch, room, splits):
    assert engine(D, batch, room, kv_bits=kv_bits).nsplit == splits
