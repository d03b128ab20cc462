"""Host side of the Llama layers' calls: what reaches the library and what is refused, on CPU tensors with the library stubbed."""
import ctypes

import pytest
import torch

from proxy_inference_engine_b200 import ops


def _bf16(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16)


def test_one_key_may_be_a_view_and_a_copy(monkeypatch):
    """One token without a cache: rotated keys are a copy, values a view of the projection's rows.  They differ in the stride of a
    dimension of one element, which says nothing; any other difference is refused."""
    H, D = 2, 64
    monkeypatch.setattr(ops._lib, "load", lambda: None)
    monkeypatch.setattr(ops, "decode_attention", lambda q, *a, **k: torch.zeros(q.shape[0], q.shape[1] * q.shape[2]))
    view = lambda B, width: _bf16(B, 1, width)[..., :H * D].reshape(B, 1, H, D).transpose(1, 2)
    for B, width in ((1, H * D), (1, 3 * H * D), (3, H * D)):
        q, k, v = _bf16(B, H, 1, D), _bf16(B, H, 1, D), view(B, width)
        assert k.stride() != v.stride()
        assert ops.scaled_dot_product_attention(q, k, v, scale=1.0).shape == (B, H, 1, D)
    with pytest.raises(ValueError, match="one layout"):   # rows of another width: the batch stride counts
        ops.scaled_dot_product_attention(q, k, view(3, 3 * H * D), scale=1.0)
    with pytest.raises(ValueError, match="one layout"):
        ops.scaled_dot_product_attention(_bf16(1, H, 1, D), _bf16(1, H, 5, D), _bf16(1, 5, H, D).transpose(1, 2), scale=1.0)


class _Expired:
    """A library one of whose waits has expired: its word reaches the host as the real one's does, once the copy has landed."""

    def __init__(self):
        self.word, self.posts = 0, []

    def pie_pipeline_words(self, words, stream):
        self.posts.append(ctypes.cast(words, ctypes.POINTER(ctypes.c_uint)))
        return 0
    pieh_pipeline_words = pie_pipeline_words

    def pie_pipeline_error(self):
        return self.word
    pieh_pipeline_error = pie_pipeline_error

    def land(self):
        for p in self.posts:
            p[0] = self.word
        self.posts.clear()


@pytest.fixture
def expired(monkeypatch):
    lib = _Expired()
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops._lib, "load", lambda: lib)
    return lib


def test_an_expired_wait_is_raised_once_its_copy_has_landed(expired):
    watch = ops.PipelineWatch(expired, "pie", page_locked=False)
    watch.check()
    expired.word = 1
    watch.post()
    watch.check()                       # nothing is waited for
    expired.land()
    for _ in range(2):                  # the word lasts, for other engines too, until it is cleared
        with pytest.raises(RuntimeError, match="expired"):
            watch.check()
    expired.word = 0
    watch.check()
    watch.post(), expired.land()
    watch.check()
    ops.check_pipeline()
    expired.word = 1
    with pytest.raises(RuntimeError, match="expired"):
        ops.check_pipeline()


def test_the_decode_engine_raises_instead_of_handing_out_void_tokens(expired):
    from proxy_inference_engine_b200.decode import DecodeEngine
    eng = object.__new__(DecodeEngine)
    eng.watch = ops.PipelineWatch(expired, "pie", page_locked=False)
    eng.positions, eng.seq, eng.prompt_len = torch.tensor([3]), torch.arange(8)[None], 2
    eng._next_pos, eng.max_context = 3, 8
    eng.watch.post(), expired.land()
    assert eng.generated().tolist() == [[2, 3]]
    for call in (eng.generated, eng.step, lambda: eng.prefill(torch.zeros(1, 4))):
        expired.word = 1
        eng.watch.post(), expired.land()
        with pytest.raises(RuntimeError, match="expired"):
            call()


def test_the_hybrid_engine_raises_at_the_end_of_a_step_and_before_the_next(expired):
    from proxy_inference_engine_b200.engine import HybridEngine

    class Model:
        device, layers = "cpu", []

        def make_cache(self, max_tokens, max_seqs):
            from proxy_inference_engine_b200.cache import HybridCache
            return HybridCache([], max_tokens, max_seqs, device="cpu", lib=ops._lib.load_hybrid(build_if_missing=True))

        def step(self, batch, cache, rows=None, trace=None):
            expired.word = int(batch.total_tokens_in_step > 2)
            return torch.zeros(len(rows), 5)

    def sampler(logits):
        expired.land()                  # the host waits for the step
        return logits.argmax(-1)

    eng = HybridEngine(Model(), max_tokens=256, max_seqs=1, use_graph=False)
    eng.watch = ops.PipelineWatch(expired, "pieh", page_locked=False)
    assert eng.generate([[1, 2]], max_new_tokens=2, sampler=sampler) == [[0, 0]]
    with pytest.raises(RuntimeError, match="expired"):
        eng.generate([[1, 2, 3]], max_new_tokens=2, sampler=sampler)
    eng.finish(("gen", 0))
    with pytest.raises(RuntimeError, match="expired"):
        eng.forward([("a", [1, 2, 3], None)])
    expired.word = 0                    # cleared
    eng.forward([("a", [1, 2, 3], None)])
    expired.land()
    with pytest.raises(RuntimeError, match="expired"):
        eng.check()


@pytest.mark.parametrize("rows", [1, 70])
@pytest.mark.parametrize("swapped", ["gate_proj", "up_proj", "both"])
def test_any_callable_may_stand_for_a_projection(monkeypatch, rows, swapped):
    """The fused calls step aside for a projection that is no QuantizedLinear, whatever it has or lacks."""
    from proxy_inference_engine_b200 import llama, nn
    K, N = 512, 256
    plain = object.__new__(nn.QuantizedLinear)
    plain.group_size, plain.bits = 64, 4
    plain.weight, plain.scales, plain.biases = torch.zeros((N, K // 8), dtype=torch.int32), _bf16(N, K // 64), _bf16(N, K // 64)
    monkeypatch.setattr(nn.QuantizedLinear, "__call__", lambda self, x: x[..., :N])
    monkeypatch.setattr(ops, "qmm_swiglu_pays", lambda *a: True)
    monkeypatch.setattr(ops, "silu_mul", lambda a, b: a + b)
    mlp = object.__new__(llama.MLP)
    mlp.down_proj = lambda a: a
    other = lambda x: x[..., :N]
    mlp.gate_proj = plain if swapped == "up_proj" else other
    mlp.up_proj = plain if swapped == "gate_proj" else other
    x = torch.ones((rows, K), dtype=torch.bfloat16)
    assert torch.equal(mlp(x), 2 * x[..., :N])


def _plain(N=256, K=512, bits=4):
    from proxy_inference_engine_b200 import nn
    lin = object.__new__(nn.QuantizedLinear)
    lin.group_size, lin.bits = 64, bits
    lin.weight, lin.scales, lin.biases = torch.zeros((N, K * bits // 32), dtype=torch.int32), _bf16(N, K // 64), _bf16(N, K // 64)
    return lin


def _with(lin, **fields):
    for name, value in fields.items():
        setattr(lin, name, value)
    return lin


def test_fused_rows_takes_what_its_kernel_takes_and_nothing_else(monkeypatch):
    from proxy_inference_engine_b200 import nn
    monkeypatch.setattr(ops, "qmv_fused", lambda *a: "fused")
    norm = object.__new__(nn.RMSNorm)
    norm.weight, norm.eps = _bf16(512), 1e-5
    x = _bf16(32, 512)
    takes = lambda x=x, lins=(_plain(),), **kw: nn.fused_rows(x, lins, **kw) == "fused"
    assert takes() and takes(_bf16(1, 1, 512)) and takes(lins=(_plain(7), _plain(300)), norm=norm)
    assert takes(residual=_bf16(32, 256)) and takes(lins=(_plain(), _plain()), swiglu=True)
    assert takes(_bf16(4, 384), (_plain(K=384, bits=8),))
    assert not takes(_bf16(33, 512)) and not takes(_bf16(0, 512))                       # rows
    assert not takes(x.float()) and not takes(_bf16(32, 1024)[:, ::2]) and not takes(_bf16(513)[1:].view(1, 512))   # type, stride, alignment
    assert not takes(_bf16(4, 384), (_plain(K=384),))                                   # K in whole stages: 256 at 4 bits, 128 at 8
    assert not takes(_bf16(4, 1024))                                                    # K of x and of the matrix
    assert not takes(lins=(_plain(), _plain(bits=8))) and not takes(lins=(_with(_plain(), group_size=32),))
    assert not takes(lins=(_with(_plain(), bias=_bf16(256)),)) and not takes(lins=(_with(_plain(), scales=torch.zeros(256, 8)),))
    other = object.__new__(type("Other", (nn.QuantizedLinear,), {}))
    other.__dict__.update(vars(_plain()))
    assert not takes(lins=(other,)) and not takes(lins=(_plain(), lambda x: x))         # a subclass may compute something else
    assert not takes(lins=(_plain(128), _plain(256)), swiglu=True)                      # halves of one width
    assert not takes(residual=_bf16(32, 255)) and not takes(residual=torch.zeros(32, 256))
    norm.weight = torch.zeros(512)
    assert not takes(norm=norm) and not takes(norm=lambda x: x)


def test_a_tensor_parallel_block_takes_the_separate_calls(monkeypatch):
    from types import SimpleNamespace
    from proxy_inference_engine_b200 import llama, nn
    monkeypatch.setattr(nn, "fused_rows", lambda *a, **k: pytest.fail("fused"))
    block = object.__new__(llama.TransformerBlock)
    block.self_attn, block.mlp = object.__new__(llama.Attention), object.__new__(llama.MLP)
    block.self_attn.tp = SimpleNamespace(on=True)
    assert block._few_rows(_bf16(1, 1, 512), None, None) is None
    block.self_attn.tp = None
    block.mlp = lambda x: x
    assert block._few_rows(_bf16(1, 1, 512), None, None) is None


@pytest.mark.parametrize("odd", [None, "bits", "wrapped"])
def test_a_prompt_layer_norms_its_input_once(monkeypatch, odd):
    """... whether or not its q, k and v go in one launch, and with the sums of the separate calls where they do not."""
    from proxy_inference_engine_b200 import llama, nn
    calls = []
    monkeypatch.setattr(nn.RMSNorm, "__call__", lambda self, x: calls.append("norm") or x)
    monkeypatch.setattr(nn.QuantizedLinear, "__call__", lambda self, x: calls.append("linear") or _bf16(*x.shape[:-1], self.weight.shape[0]))
    monkeypatch.setattr(ops, "qmm_rows", lambda x, lins, rows, K, N, residual: calls.append(len(lins)) or _bf16(*x.shape[:-1], N))
    monkeypatch.setattr(ops, "qmm_swiglu_pays", lambda *a: False)
    monkeypatch.setattr(ops, "silu_mul", lambda g, u: g)
    monkeypatch.setattr(ops, "add", lambda a, b: a + b)
    monkeypatch.setattr(llama.Attention, "attend", lambda self, q, k, v, B, L, mask, cache: _bf16(B, L, q.shape[-1]))
    at, mlp = object.__new__(llama.Attention), object.__new__(llama.MLP)
    at.q_proj, at.k_proj, at.v_proj, at.o_proj = _plain(512), _plain(256), _plain(256), _plain(512)
    mlp.gate_proj, mlp.up_proj, mlp.down_proj = _plain(512), _plain(512), _plain(512)
    if odd == "bits":
        at.v_proj = _plain(256, bits=8)
    if odd == "wrapped":
        at.k_proj = lambda x, inner=at.k_proj: inner(x)
    layer = object.__new__(llama.TransformerBlock)
    layer.self_attn, layer.mlp = at, mlp
    layer.input_layernorm, layer.post_attention_layernorm = object.__new__(nn.RMSNorm), object.__new__(nn.RMSNorm)
    x = _bf16(1, 200, 512)
    assert layer(x).shape == x.shape and calls.count("norm") == 2
    assert calls == ["norm"] + ([3] if odd is None else ["linear"] * 3) + [1, "norm", "linear", "linear", 1]


class _Rows:
    """Projected rows as a GPU has them."""
    is_cuda = True

    def __getitem__(self, at):
        return self


@pytest.mark.parametrize("where", ["nowhere", "object", "class", "cache", "cache's class"])
def test_a_decode_step_calls_what_is_put_in_a_methods_place(where, monkeypatch):
    """... on one attention object or cache, or on its class: the native call is for the methods that it stands for."""
    from types import SimpleNamespace
    from proxy_inference_engine_b200 import llama
    from proxy_inference_engine_b200.cache import KVCache
    monkeypatch.setattr(ops, "native_host", lambda: SimpleNamespace(attend_rows=lambda *a: "native"))
    at, cache = object.__new__(llama.Attention), KVCache()
    at.q_proj, at.k_proj, at.v_proj = _plain(512), _plain(256), _plain(256)
    theirs = lambda *a: "theirs"
    if where != "nowhere":
        monkeypatch.setattr(*{"object": (at, "attend"), "class": (llama.Attention, "attend"), "cache": (cache, "update_and_fetch"),
                              "cache's class": (KVCache, "update_and_fetch")}[where], theirs, raising=False)
    if where.startswith("cache"):
        assert not llama._rotates(cache)
        monkeypatch.setattr(at, "attend", theirs, raising=False)
    assert at.attend_beside(_Rows(), torch.zeros((2, 1, 512)), None, cache) == ("native" if where == "nowhere" else "theirs")


def test_a_host_module_that_does_not_load_leaves_the_calls_to_python(monkeypatch):
    """... as one that was built for another torch or interpreter does: a warning, once, and no answer to any call."""
    def refuse(*args):
        raise ImportError("undefined symbol")
    ops.native_fused_rows.cache_clear()
    try:
        with monkeypatch.context() as m:
            m.setattr(ops.os.path, "exists", lambda path: True)
            m.setattr(ops.importlib.util, "module_from_spec", refuse)
            with pytest.warns(UserWarning, match="does not load"):
                assert ops.native_fused_rows()(1, 2, 3) is None
            assert ops.native_fused_rows()(1, 2, 3) is None
    finally:
        ops.native_fused_rows.cache_clear()


def _four_addresses(a, b, c, d):
    pass


@pytest.mark.parametrize("old", [dict(bind=_four_addresses), dict(bind=_four_addresses, functions=["pie_qmt"]), dict(functions=["pie_no_such_call"]),
                                 dict(functions=[], bind=lambda table: {}["pie_qmt"]), dict(functions=[], bind=lambda table: None, fused_rows=lambda *a: 1)])
def test_a_host_module_of_another_build_leaves_the_calls_to_python(old, monkeypatch):
    """It loads, but wants other functions of the library, is bound in another way, or has fewer calls."""
    from types import SimpleNamespace
    spec = SimpleNamespace(loader=SimpleNamespace(exec_module=lambda host: None))
    ops.native_fused_rows.cache_clear()
    try:
        with monkeypatch.context() as m:
            m.setattr(ops.os.path, "exists", lambda path: True)
            m.setattr(ops.importlib.util, "spec_from_file_location", lambda *a: spec)
            m.setattr(ops.importlib.util, "module_from_spec", lambda spec: SimpleNamespace(**old))
            with pytest.warns(UserWarning, match="does not load"):
                assert ops.native_fused_rows()(1, 2, 3) is None
            assert ops.native_host().mlp_rows(1, 2) is None and ops.native_host().attend_rows(1, 2) is None
    finally:
        ops.native_fused_rows.cache_clear()


def test_the_matmuls_route_is_asked_for_at_every_call(monkeypatch):
    """PIE_QMT and the current device may change between two calls: the Python form answers as the library, and so as the native form, does."""
    answers = []
    for mode in ("2", "0", "2"):
        monkeypatch.setenv("PIE_QMT", mode)
        answers.append(ops.qmt_scratch_bytes(40, 2048, 2048, 4, 0))
    assert answers[0] == answers[2] > 0 == answers[1]
