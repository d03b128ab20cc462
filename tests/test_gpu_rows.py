"""Layers of few rows in native calls, and rotation and cache write in one launch: the bits of the separate calls."""
import pytest
import torch

from parity_util import tiny_args

pytestmark = pytest.mark.gpu


def _heads(g, B, H, L, D, order):
    """[B, H, L, D] bf16 as projections leave it: its own rows (beside others in wider rows), or contiguous."""
    if order == "own":
        return torch.randn((B, H, L, D), generator=g, device="cuda").bfloat16()
    wide = torch.randn((B, L, H * D + (8 if order == "beside" else 3)), generator=g, device="cuda").bfloat16()
    return wide[..., :H * D].unflatten(-1, (H, D)).transpose(1, 2)


def _caches(kind, B, H, D, room, g):
    from proxy_inference_engine_b200 import cache as C
    table = torch.randperm(B * ((room + 63) // 64), generator=torch.Generator().manual_seed(room)).to(torch.int32).view(B, -1).cuda()
    pool = lambda: torch.zeros((table.numel(), 64, H, D), dtype=torch.bfloat16, device="cuda")
    make = {"plain": lambda: C.KVCache(room), "paged": lambda: C.PagedKVCache(pool(), pool(), table), "quantized": lambda: C.QuantizedKVCache(64, 8, room),
            "paged quantized": lambda: C.PagedQuantizedKVCache(table.numel(), H, D, table)}[kind]
    return make(), make()


def _contents(c):
    from proxy_inference_engine_b200.cache import PagedKVCache, PagedQuantizedKVCache, QuantizedKVCache
    if isinstance(c, PagedKVCache):
        return [c.k_pool, c.v_pool]
    if isinstance(c, (QuantizedKVCache, PagedQuantizedKVCache)):
        return [*c.keys, *c.values]
    return [c.keys, c.values]


@pytest.mark.parametrize("kind", ["plain", "paged", "quantized", "paged quantized"])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("order", ["own", "beside", "odd"])      # odd: rows that are not 16-byte aligned
@pytest.mark.parametrize("B,L,past", [(1, 1, 0), (5, 1, 130), (1, 48, 7), (1, 49, 7), (3, 40, 64), (2, 700, 61), (1, 768, 0), (1, 769, 0)])
def test_rotation_and_cache_write_in_one_launch(kind, D, order, B, L, past):
    from proxy_inference_engine_b200.llama import Llama3RoPE
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + L + D)
    Hq, Hkv = 8, 2
    rope = Llama3RoPE(131072, 131072, D, 500000.0, 8.0, 1.0, 4.0)
    one, two = _caches(kind, B, Hkv, D, past + L, g)
    if past:
        old = [torch.randn((B, Hkv, past, D), generator=g, device="cuda").bfloat16() for _ in "kv"]
        for c in (one, two):
            c.update_and_fetch(*old)
    q, k, v = (_heads(g, B, H, L, D, order) for H in (Hq, Hkv, Hkv))
    got = one.rotate_and_fetch(q, k, v, rope._freqs)
    if "quantized" in kind and B * L * (Hq + 2 * Hkv) > 9216:
        assert got is None and one.offset == past
        return
    want = rope(q, offset=past)
    two.update_and_fetch(rope(k, offset=past), v)
    assert got[0].is_contiguous() and torch.equal(got[0], want) and one.offset == two.offset == past + L
    assert all(torch.equal(a, b) for a, b in zip(_contents(one), _contents(two)))


def test_a_full_page_table_is_refused():
    from proxy_inference_engine_b200.llama import Llama3RoPE
    g = torch.Generator(device="cuda").manual_seed(1)
    rope = Llama3RoPE(131072, 131072, 64, 500000.0, 8.0, 1.0, 4.0)
    for kind in ("paged", "paged quantized"):
        c, _ = _caches(kind, 1, 2, 64, 64, g)
        with pytest.raises(ValueError, match="page table too small"):
            c.rotate_and_fetch(*(_heads(g, 1, H, 65, 64, "own") for H in (4, 2, 2)), rope._freqs)
        assert c.offset == 0


def _block(bits, D, seed=0):
    from proxy_inference_engine_b200.checkpoint import build_model, random_weights
    args = tiny_args(bits=bits, head_dim=D, hidden_size=512, intermediate_size=1024, num_attention_heads=8, num_key_value_heads=2, num_hidden_layers=1)
    return build_model(args, random_weights(args, seed=seed, device="cuda")).layers[0]


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kv", [None, 8])
@pytest.mark.parametrize("B", [1, 2, 8, 9, 32, 33])          # either side of the matmuls' row counts
def test_a_decode_steps_layer_is_the_python_forms(bits, D, kv, B, monkeypatch):
    from proxy_inference_engine_b200 import ops
    from proxy_inference_engine_b200.cache import KVCache, QuantizedKVCache
    g, block = torch.Generator(device="cuda").manual_seed(B + D), _block(bits, D)
    old = [torch.randn((B, 2, 300, D), generator=g, device="cuda").bfloat16() for _ in "kv"]
    xs = [torch.randn((B, 1, 512), generator=g, device="cuda").bfloat16() for _ in range(3)]
    outs, caches = [], []
    for native in (True, False):
        cache = KVCache(303) if kv is None else QuantizedKVCache(64, 8, 303)
        cache.update_and_fetch(*old)
        with monkeypatch.context() as m:
            if not native:
                m.setattr(ops, "native_fused_rows", lambda: lambda *a: None)
            outs.append([block(x, None, cache) for x in xs])
        caches.append(cache)
    assert caches[0].offset == caches[1].offset == 303
    assert all(torch.equal(a, b) for a, b in zip(outs[0], outs[1]))
    assert all(torch.equal(a, b) for a, b in zip(_contents(caches[0]), _contents(caches[1])))


def test_a_decode_steps_layer_goes_as_far_as_it_can(monkeypatch):
    """A cache that has to grow, a biased projection, a wrapped one, a rotation that is not its own: the Python form goes on from there."""
    from proxy_inference_engine_b200 import nn, ops
    from proxy_inference_engine_b200.cache import KVCache
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((2, 1, 512), generator=g, device="cuda").bfloat16()

    def call(change):
        outs = []
        for native in (True, False):
            block, cache = _block(4, 64), KVCache()
            cache.update_and_fetch(*(torch.randn((2, 2, 256, 64), generator=torch.Generator(device="cuda").manual_seed(4), device="cuda").bfloat16() for _ in "kv"))
            change(block, cache)
            with monkeypatch.context() as m:
                if not native:
                    m.setattr(ops, "native_fused_rows", lambda: lambda *a: None)
                outs += [block(x, None, cache), cache.keys, cache.values, torch.tensor(cache.offset)]
        assert all(torch.equal(a, b) for a, b in zip(outs[:4], outs[4:])) and int(outs[3]) == 257

    def biased(name, part):
        def change(block, cache):
            cache.reserve(2, 2, 64, 257)
            getattr(getattr(block, part), name).bias = torch.ones((), dtype=torch.bfloat16, device="cuda")
        return change

    def wrapped(block, cache):
        cache.reserve(2, 2, 64, 257)
        inner = block.self_attn.o_proj
        block.self_attn.o_proj = lambda v: inner(v)

    class Rope:
        def __init__(self, rope): self.rope = rope
        def __call__(self, v, offset=0): return self.rope(v, offset=offset)

    def other_rope(block, cache):
        cache.reserve(2, 2, 64, 257)
        block.self_attn.rope = Rope(block.self_attn.rope)

    call(lambda block, cache: None)                              # 256 rows are full: it grows
    for name, part in (("q_proj", "self_attn"), ("o_proj", "self_attn"), ("gate_proj", "mlp"), ("down_proj", "mlp")):
        call(biased(name, part))
    call(wrapped)
    call(other_rope)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("rows", [1, 3, 8, 9, 20, 32, 40, 100])
def test_a_feed_forward_of_few_rows_is_the_python_forms(bits, rows, monkeypatch):
    from proxy_inference_engine_b200 import ops
    g, mlp = torch.Generator(device="cuda").manual_seed(rows), _block(bits, 64).mlp
    x = torch.randn((rows, 512), generator=g, device="cuda").bfloat16()
    outs = [mlp(x) for _ in range(3)]                            # (the second launch of each runs ahead of the end of the first)
    with monkeypatch.context() as m:
        m.setattr(ops, "native_fused_rows", lambda: lambda *a: None)
        want = mlp(x)
    assert all(torch.equal(y, want) for y in outs)


def test_a_layer_on_a_stream_of_its_own_and_in_a_capture():
    from proxy_inference_engine_b200.cache import KVCache
    g, block = torch.Generator(device="cuda").manual_seed(6), _block(4, 128)
    old = [torch.randn((2, 2, 100, 128), generator=g, device="cuda").bfloat16() for _ in "kv"]
    x = torch.randn((2, 1, 512), generator=g, device="cuda").bfloat16()

    def step(v):
        cache = KVCache(101)
        cache.update_and_fetch(*old)
        return block(v, None, cache)

    want, twice, side = step(x), step(2 * x), torch.cuda.Stream()
    a = torch.randn((8192, 8192), device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        late = x * 0
        for _ in range(3):
            torch.mm(a, a)
        late.copy_(x)
        got = step(late)
    side.synchronize()
    assert torch.equal(got, want)
    graph, fed = torch.cuda.CUDAGraph(), x.clone()
    with torch.cuda.graph(graph):
        out = step(fed)
    for v, y in ((x, want), (2 * x, twice), (x, want)):
        fed.copy_(v)
        graph.replay()
        assert torch.equal(out, y)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("rows", [1, 4, 9, 40, 200])
@pytest.mark.parametrize("written", ["gate_proj", "up_proj", "down_proj"])
def test_weights_written_by_the_launch_before(bits, rows, written):
    """Launches set themselves up, and ask L2 for weights, under the end of the launch before them: what that one writes into the weights is what they multiply by.
    It is a norm of one long row, a single block that lets its dependents start at its top and writes a matrix's scales last of all."""
    from proxy_inference_engine_b200 import _lib
    L = _lib.load()
    g, mlp = torch.Generator(device="cuda").manual_seed(rows), _block(bits, 64).mlp
    x = torch.randn((rows, 512), generator=g, device="cuda").bfloat16()
    lin, long = getattr(mlp, written), 1 << 18
    out, ones, n = torch.ones(long, device="cuda").bfloat16(), torch.ones(long, device="cuda").bfloat16(), lin.scales.numel()
    sets = []                                                    # a norm of ones is its weight
    for i in range(2):
        sets.append(ones.clone())
        sets[i][long - n:] = lin.scales.flatten() * (1 + 2 * i)
    lin.scales = out[long - n:].view(lin.scales.shape)
    want = []
    for w in sets:
        out.copy_(w)
        torch.cuda.synchronize()
        want.append(mlp(x))
    assert not torch.equal(*want)
    got = []
    for i in range(20):
        assert L.pie_rms_norm(out.data_ptr(), ones.data_ptr(), sets[i % 2].data_ptr(), 1, long, 0.0, torch.cuda.current_stream().cuda_stream) == 0
        got.append(mlp(x))
    assert torch.equal(out, sets[1]) and all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))
