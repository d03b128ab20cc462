"""How many parts decode attention cuts a context into, for heads of 64."""
import pytest

from proxy_inference_engine_b200 import _lib


@pytest.mark.parametrize("heads", [(32, 8), (6, 2), (16, 1), (17, 1), (40, 2), (8, 8)])
@pytest.mark.parametrize("B", [0, 1, 2, 5, 8, 16, 32, 75, 600])
@pytest.mark.parametrize("ctx", [1, 64, 127, 128, 500, 1066, 2048, 7002, 100000])
def test_heads_of_64_may_have_more_splits(heads, B, ctx):
    """Never fewer than for heads of 128, which keep theirs; more only while a split has 128 tokens and four CTAs an SM hold all of them."""
    L = _lib.load()
    few, more = (L.pie_decode_attn_pick_splits_for(B, *heads, d, ctx) for d in (128, 64))
    assert few == L.pie_decode_attn_pick_splits(B, *heads, ctx)
    assert more >= few
    if more > few:
        assert heads[0] // heads[1] <= 16 and more <= 32 and ctx // more >= 128 and B * heads[1] * more <= 4 * 148
