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


@pytest.mark.parametrize("B,ctx,splits", [(1, 383, 1), (1, 384, 3), (8, 383, 1), (8, 450, 2), (10, 799, 1), (16, 799, 1), (16, 800, 2), (16, 1300, 2), (75, 9000, 1), (1, 8192, 16)])
def test_8_bit_splits_only_where_their_sum_pays(B, ctx, splits):
    """Two of 128 tokens, or two on one SM below 400 each, measured slower than one."""
    assert _lib.load().pie_decode_attn_q8_pick_splits(B, 32, 8, ctx) == splits


@pytest.mark.parametrize("B,ctx,splits", [(32, 383, 1), (32, 384, 2), (4, 1300, 9), (8, 640, 5), (4, 1536, 12), (16, 384, 3)])
def test_heads_of_64_have_more_splits_only_where_that_pays(B, ctx, splits):
    """A first sum of splits, and one split more of nine, measured slower."""
    assert _lib.load().pie_decode_attn_pick_splits_for(B, 32, 8, 64, ctx) == splits


@pytest.mark.parametrize("B,Hkv", [(1 << 16, 1 << 16), (1 << 15, 1 << 16), (1 << 30, 8), ((1 << 31) - 1, 2)])
def test_more_heads_than_32_bits_count(B, Hkv):
    """(a product of 2^32 was a division by zero)"""
    L = _lib.load()
    for D in (64, 128):
        assert L.pie_decode_attn_pick_splits_for(B, Hkv, Hkv, D, 4096) == 1
    assert L.pie_decode_attn_q8_pick_splits(B, Hkv, Hkv, 4096) == 1
