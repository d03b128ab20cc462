"""The tcgen05 tile kernels (pie_gemm.cuh: quantized prefill GEMM and dense linear; pie_fa_prefill.cu) against float64, at the
edges of their tiles and on every route of their dispatch.  The bounds are elementwise and derived: a result rounded once to
bf16 (8 significant bits) is off by at most 2^-8 of itself; an fp32 sum of K products by at most K 2^-24 of the sum of their magnitudes (2^-23
where the tensor core truncates instead of rounding)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _within(got, want, slack):
    off = (got.double() - want).abs() - slack
    assert torch.isfinite(got).all() and off.max() <= 0, float(off.max())


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,N,K", [(64, 128, 128),        # one tile, one packed chunk that is not full (4 bits)
                                   (77, 300, 384),        # ragged rows and columns, scales one at a time
                                   (129, 257, 512),       # one past a tile both ways, scales eight at a time
                                   (70, 640, 14336),      # K over four ranks of a cluster
                                   (200, 1024, 1152),     # a last rank with fewer steps
                                   (513, 4100, 640),      # more tiles than one wave of single CTAs
                                   (2050, 2056, 1024),    # CTA pairs, ragged both ways, several tiles a pair
                                   (1000, 14336, 128),    # pairs of 224 columns
                                   (1500, 2100, 1024),    # pairs of 192
                                   (400, 3000, 256)])     # pairs of 128
def test_quantized_gemm_tiles(bits, M, N, K):
    from proxy_inference_engine_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K + bits)
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    wq, s, b = ops.quantize(w, 64, bits)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    shifts = torch.arange(0, 32, bits, device="cuda", dtype=torch.int32)
    q = ((wq[:, :, None] >> shifts) & (2 ** bits - 1)).reshape(N, K // 64, 64).double()
    dense = (q * s.double()[:, :, None] + b.double()[:, :, None]).reshape(N, K).to(torch.bfloat16).double()
    want, mass = x.double() @ dense.t(), x.double().abs() @ dense.abs().t()
    # w_hat comes from fp32 (8 bits) or a fused bf16 operation: where the float64 value sits on a rounding boundary it may
    # differ by an ulp, up to 2^-7 of the weight, in a few weights of a thousand: allow 2^-7 / 256 of the mass
    _within(ops.quantized_matmul(x, wq, s, b, group_size=64, bits=bits), want, want.abs() * 2 ** -8 + mass * (K * 2 ** -23 + 2 ** -15))
    assert _lib.load().pie_pipeline_error() == 0


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,N,K", [(64, 128, 128),        # 128 columns a tile pair, 64 of y; one tile
                                   (300, 1100, 384),      # the same, ragged
                                   (1500, 2100, 1024),    # 192
                                   (777, 4100, 640),      # 256, rows of y off 16 bytes, scales one at a time
                                   (2050, 2056, 1024)])   # several tiles a pair
def test_swiglu_in_the_gemm_is_the_separate_operators(bits, M, N, K):
    """Both products sum K in the order of the separate ones and every rounding is kept: the same bits."""
    from proxy_inference_engine_b200 import _lib, nn, ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K + bits)
    lins = []
    for _ in range(2):
        lin = nn.QuantizedLinear(K, N, bias=False, group_size=64, bits=bits)
        lin.weight, lin.scales, lin.biases = ops.quantize(torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16), 64, bits)
        lins.append(lin)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    got = nn.fused_swiglu(x, *lins)
    assert got is not None and torch.equal(got, ops.silu_mul(lins[0](x), lins[1](x)))
    assert nn.fused_swiglu(x[:63], *lins) is None and nn.fused_swiglu(x.float(), *lins) is None
    assert _lib.load().pie_pipeline_error() == 0


@pytest.mark.parametrize("M,N,K", [(33, 64, 64), (129, 257, 128), (70, 640, 8192), (200, 1024, 1152), (513, 4100, 192), (2050, 2056, 512), (1200, 8192, 128),
                                   (700, 3000, 128)])
def test_dense_gemm_tiles(M, N, K):
    from proxy_inference_engine_b200 import _lib
    L = _lib.load_hybrid(build_if_missing=True)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    want = x.double() @ w.double().t()
    slack = (x.double().abs() @ w.double().abs().t()) * (K * 2 ** -23)
    for dt, code, rel in ((torch.float32, 1, 0.0), (torch.bfloat16, 0, 2 ** -8)):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=dt)
        assert L.pieh_linear(_p(out), code, N, _p(x), 0, K, _p(w), 0, None, M, N, K, 0, 0.0, None, None, 0, None) == 0
        _within(out, want, slack + want.abs() * rel)
    for S in (1, 2, 3, 4):   # the residual-stream update: one routine for 1, 2 and 4 streams, another for the rest
        xs = torch.randn((M, S, N), generator=g, device="cuda")
        mix, ow = torch.randn((S, S), generator=g, device="cuda"), torch.randn((S,), generator=g, device="cuda")
        ref = torch.einsum("su,msn->mun", mix.double(), xs.double()) + ow.double()[None, :, None] * want[:, None]
        size = torch.einsum("su,msn->mun", mix.double().abs(), xs.double().abs()) + ow.double().abs()[None, :, None] * want.abs()[:, None]
        assert L.pieh_linear(_p(xs), 1, 0, _p(x), 0, K, _p(w), 0, None, M, N, K, 3, 0.0, _p(mix), _p(ow), S, None) == 0
        _within(xs, ref, size * (2 * S * 2 ** -23) + ow.double().abs()[None, :, None] * slack[:, None])
    assert L.pieh_pipeline_error() == 0


@pytest.mark.parametrize("step", [0, -1])   # rows that repeat, rows that go backward
def test_dense_rows_a_tiled_copy_cannot_describe(step):
    from proxy_inference_engine_b200 import _lib
    L = _lib.load_hybrid(build_if_missing=True)
    g = torch.Generator(device="cuda").manual_seed(5)
    M, N, K = 70, 130, 128
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    rows = x.flip(0) if step else x[-1:].expand(M, K)
    out = torch.full((M, N), float("nan"), device="cuda")
    assert L.pieh_linear(_p(out), 1, N, _p(x[-1]), 0, step * K, _p(w), 0, None, M, N, K, 0, 0.0, None, None, 0, None) == 0
    _within(out, rows.double() @ w.double().t(), (rows.double().abs() @ w.double().abs().t()) * (K * 2 ** -23))


@pytest.mark.parametrize("shared", ["", "x", "w"])
def test_dense_gemm_batched(shared):
    """Products side by side, head-major columns; an operand stride of zero shares that operand."""
    from proxy_inference_engine_b200 import _lib
    L = _lib.load_hybrid(build_if_missing=True)
    g = torch.Generator(device="cuda").manual_seed(3)
    M, N, K, nb = 150, 72, 128, 5
    x = torch.randn((M, nb, K), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn((nb, N, K), generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M, nb, N), float("nan"), device="cuda")
    assert L.pieh_linear_batched(_p(out), 1, nb * N, N, _p(x), 0, nb * K, 0 if shared == "x" else K, _p(w), 0,
                                 0 if shared == "w" else N * K, nb, M, N, K, 0, None, 0, 0, None) == 0
    xr = (x[:, :1].expand(M, nb, K) if shared == "x" else x).double()
    wr = (w[:1].expand(nb, N, K) if shared == "w" else w).double()
    want = torch.einsum("mzk,znk->mzn", xr, wr)
    _within(out, want, torch.einsum("mzk,znk->mzn", xr.abs(), wr.abs()) * (K * 2 ** -23))


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,offset", [(1, 2, 1, 1, 0),        # one query, one key
                                               (1, 2, 2, 2, 255),      # two queries across a key tile's end
                                               (2, 4, 2, 129, 0),      # one row in the second query tile
                                               (1, 4, 1, 256, 128),    # whole tiles
                                               (2, 4, 2, 300, 77),     # ragged everywhere
                                               (1, 2, 1, 1030, 517)])  # several blocks, the ring wraps
def test_prefill_attention_tiles(paged, D, B, Hq, Hkv, L, offset):
    from proxy_inference_engine_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(L + offset + D)
    T, scale = offset + L, D ** -0.5
    rnd = lambda *s: (1.5 * torch.randn(s, generator=g, device="cuda")).to(torch.bfloat16)
    q, k, v = rnd(B, Hq, L, D), rnd(B, Hkv, T, D), rnd(B, Hkv, T, D)
    nan = float("nan")   # slots no token was written to: what is there must not matter
    if paged:
        n = (T + 63) // 64
        kb, vb = (torch.full((B * n + 2, 64, Hkv, D), nan, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        table = torch.full((B, n + 1), -1, device="cuda", dtype=torch.int32)
        table[:, :n] = torch.randperm(B * n + 2, generator=g, device="cuda")[:B * n].view(B, n)
        t = torch.arange(T, device="cuda")
        for b in range(B):
            kb[table[b, t // 64].long(), t % 64], vb[table[b, t // 64].long(), t % 64] = k[b].transpose(0, 1), v[b].transpose(0, 1)
        lay = ops.kv_layout(kb, table, 64)
    else:
        kb, vb = (torch.full((B, Hkv, T + 70, D), nan, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        kb[:, :, :T], vb[:, :, :T] = k, v
        lay = ops.kv_layout(kb)
    got = ops.prefill_attention(q, kb, vb, lay, offset, scale)
    rep = Hq // Hkv
    s = torch.einsum("bhld,bhtd->bhlt", q.double(), k.double().repeat_interleave(rep, 1)) * scale
    i, j = torch.arange(L, device="cuda")[:, None] + offset, torch.arange(T, device="cuda")[None]
    p = torch.softmax(s.masked_fill(j > i, float("-inf")), -1)
    vr = v.double().repeat_interleave(rep, 1)
    want, mass = p @ vr, p @ vr.abs()
    # each weight rounded to bf16 (2^-8 of it), the result rounded once; scores are fp32 sums of D products of size |s| and the
    # exponential turns their error into a relative one
    slack = mass * (2 ** -8 + 2 * D * 2 ** -23 * float(s.abs().max())) + want.abs() * 2 ** -8
    _within(got, want, slack)
    assert _lib.load().pie_pipeline_error() == 0


@pytest.mark.parametrize("page", [0, 64, 128, 192, 48])    # 0: contiguous; 48: no whole 64-key boxes, the mma.sync kernel's
@pytest.mark.parametrize("D,B,Hq,L,offset", [(64, 1, 2, 65, 63), (64, 1, 2, 128, 190),      # either side of the rule between them: one
                                             (64, 1, 2, 128, 255), (64, 1, 2, 100, 1000),    # query tile,
                                             (64, 1, 2, 129, 511), (64, 1, 2, 129, 639),     # two,
                                             (64, 2, 64, 129, 0), (64, 2, 32, 300, 77),      # more than one wave,
                                             (64, 40, 32, 8, 128), (64, 40, 32, 128, 256),
                                             (64, 1, 2, 1, 1030), (64, 1, 2, 129, 900), (64, 1, 4, 256, 896),   # past the rule: tile edges at D 64
                                             (128, 1, 2, 64, 0), (128, 1, 2, 60, 5), (128, 2, 4, 200, 121)])
def test_prefill_attention_routes_and_pages(page, D, B, Hq, L, offset):
    """Both kernels at the edges of the rule between them, over pages of one, two and three 64-key boxes and of none; what slots without
    a token hold must not matter."""
    from proxy_inference_engine_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(L + offset + D)
    T, scale, Hkv = offset + L, D ** -0.5, 2
    rnd = lambda *s: (1.5 * torch.randn(s, generator=g, device="cuda")).to(torch.bfloat16)
    q, k, v = rnd(B, Hq, L, D), rnd(B, Hkv, T, D), rnd(B, Hkv, T, D)
    if page:
        n = (T + page - 1) // page
        kb, vb = (torch.full((B * n + 2, page, Hkv, D), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
        table = torch.full((B, n + 1), -1, device="cuda", dtype=torch.int32)
        table[:, :n] = torch.randperm(B * n + 2, generator=g, device="cuda")[:B * n].view(B, n)
        t = torch.arange(T, device="cuda")
        for b in range(B):
            kb[table[b, t // page].long(), t % page], vb[table[b, t // page].long(), t % page] = k[b].transpose(0, 1), v[b].transpose(0, 1)
        got = ops.prefill_attention(q, kb, vb, ops.kv_layout(kb, table, page), offset, scale)
    else:
        got = ops.prefill_attention(q, k, v, ops.kv_layout(k), offset, scale)
    s = torch.einsum("bhld,bhtd->bhlt", q.double(), k.double().repeat_interleave(Hq // Hkv, 1)) * scale
    i, j = torch.arange(L, device="cuda")[:, None] + offset, torch.arange(T, device="cuda")[None]
    p = torch.softmax(s.masked_fill(j > i, float("-inf")), -1)
    vr = v.double().repeat_interleave(Hq // Hkv, 1)
    want, mass = p @ vr, p @ vr.abs()
    # the bound of test_prefill_attention_tiles
    _within(got, want, mass * (2 ** -8 + 2 * D * 2 ** -23 * float(s.abs().max())) + want.abs() * 2 ** -8)
    assert _lib.load().pie_pipeline_error() == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("scale", [0.1, 4.0, 0.0, -0.1])   # exponents down to 0 and past the smallest; not positive: the other kernel
def test_prefill_attention_exponentials(D, scale):
    """Keys beyond a row weigh exactly nothing whatever lies there, a NaN key reaches every row that sees it and no other."""
    from proxy_inference_engine_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(D)
    L = 200
    rnd = lambda *s: (1.5 * torch.randn(s, generator=g, device="cuda")).to(torch.bfloat16)
    q, k, v = rnd(1, 1, L, D), rnd(1, 1, L, D), rnd(1, 1, L, D)
    k[0, 0, 180:188], v[0, 0, 188:] = float("nan"), 3e38
    rows = ops.prefill_attention(q, k, v, ops.kv_layout(k), 0, scale).reshape(L, D)
    seen = 180
    s = (q[0, 0, :seen].double() @ k[0, 0, :seen].double().T) * scale
    p = torch.softmax(s.masked_fill(torch.ones_like(s).triu(1) > 0, float("-inf")), -1)
    want, mass = p @ v[0, 0, :seen].double(), p @ v[0, 0, :seen].double().abs()
    # as above; 200 weights below the smallest fp32 number add nothing that a bound of 2^-100 would not cover
    slack = mass * (2 ** -8 + 2 * D * 2 ** -23 * float(s.abs().max())) + want.abs() * 2 ** -8 + 2 ** -100
    _within(rows[:seen], want, slack)
    for key in range(180, 188):                      # one NaN key alone
        k1 = k.clone()
        k1[0, 0, 180:188] = 0
        k1[0, 0, key] = float("nan")
        rows = ops.prefill_attention(q, k1, v, ops.kv_layout(k1), 0, scale).reshape(L, D)
        assert not rows[:key].isnan().any() and rows[key:].isnan().all(), key


@pytest.mark.parametrize("rows,dims", [(1, 8), (3, 2048), (2, 2056), (5, 4096), (3, 8192), (2, 8200), (3, 100)])
def test_row_and_elementwise_operators(rows, dims):
    """RMSNorm at the edges of its register tiles, SwiGLU and the sum with and without 16-byte alignment and a tail."""
    from proxy_inference_engine_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(dims)
    rnd = lambda *s: (3 * torch.randn(s, generator=g, device="cuda")).to(torch.bfloat16)
    x, w = rnd(rows, dims), rnd(dims)
    n = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5)
    _within(ops.rms_norm(x, w, 1e-5), n * w.double(), (n * w.double()).abs() * 2.1 * 2 ** -8)      # rounded twice
    _within(ops.rms_norm(x, None, 1e-5), n, n.abs() * 1.1 * 2 ** -8)
    a, b = rnd(rows * dims + 5), rnd(rows * dims + 5)
    for off in (0, 1):   # 1: not 16-byte aligned
        u, v = a[off:], b[off:]
        want = u.double() * torch.sigmoid(u.double()) * v.double()
        _within(ops.silu_mul(u, v), want, want.abs() * 3.1 * 2 ** -8)                              # rounded three times
        assert torch.equal(ops.add(u, v), u + v)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,L,offset", [(1, 1, 7), (3, 5, 0), (2, 513, 100)])
def test_rope_and_cache_write_of_strided_heads(D, B, L, offset):
    """Heads as the projection wrote them give the same bits as a contiguous copy of them; so does the cache."""
    from proxy_inference_engine_b200 import ops
    from proxy_inference_engine_b200.cache import KVCache
    g = torch.Generator(device="cuda").manual_seed(L + D)
    H, pad = 3, 8
    rows = torch.randn((B, L, 2 * H * D + pad), generator=g, device="cuda").to(torch.bfloat16)   # k and v side by side
    k, v = (rows[..., i * H * D:(i + 1) * H * D].reshape(B, L, H, D).transpose(1, 2) for i in (0, 1))
    freqs = torch.linspace(1.0, 500.0, D // 2, device="cuda")
    turned = ops.rope(k, D, freqs=freqs, offset=offset)
    assert torch.equal(turned, ops.rope(k.contiguous(), D, freqs=freqs, offset=offset))
    theta = (torch.arange(L, device="cuda") + offset)[:, None] / freqs.double()
    a, b = k.double().chunk(2, -1)
    want = torch.cat([a * theta.cos() - b * theta.sin(), a * theta.sin() + b * theta.cos()], -1)
    _within(turned, want, want.abs() * 2 ** -8 + 1e-5 * (1 + offset + L) ** 0.5)   # angles in fp32
    cache, plain = KVCache(offset + L), KVCache(offset + L)
    for c, kk, vv in ((cache, k, v), (plain, k.contiguous(), v.contiguous())):
        c.update_and_fetch(torch.zeros((B, H, offset, D), device="cuda", dtype=torch.bfloat16),
                           torch.zeros((B, H, offset, D), device="cuda", dtype=torch.bfloat16)) if offset else None
        c.update_and_fetch(kk, vv)
    assert torch.equal(cache.keys, plain.keys) and torch.equal(cache.values, plain.values)
    assert torch.equal(cache.values[:, :, offset:offset + L], v)


@pytest.mark.parametrize("M,N,K", [(1, 16, 8), (4, 17, 72), (8, 300, 520), (9, 40, 1000), (32, 130, 2048)])
def test_dense_matmul_of_few_rows(M, N, K):
    """bf16 activations and weights, up to 32 rows (linear_rows_mma_kernel), plain and gated-pair epilogues."""
    from proxy_inference_engine_b200 import _lib
    L = _lib.load_hybrid(build_if_missing=True)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn((M, K + 8), generator=g, device="cuda").to(torch.bfloat16)[:, :K]     # rows further apart than they are long
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    want = x.double() @ w.double().t()
    slack = (x.double().abs() @ w.double().abs().t()) * (K * 2 ** -23)
    for dt, code, rel in ((torch.float32, 1, 0.0), (torch.bfloat16, 0, 2 ** -8)):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=dt)
        assert L.pieh_linear(_p(out), code, N, _p(x), 0, K + 8, _p(w), 0, None, M, N, K, 0, 0.0, None, None, 0, None) == 0
        _within(out, want, slack + want.abs() * rel)
    if N % 2 == 0:
        out = torch.full((M, N // 2), float("nan"), device="cuda")
        assert L.pieh_linear_glu(_p(out), 1, N // 2, _p(x), 0, K + 8, _p(w), 0, M, N, K, 1.0, 0.0, 0.0, None) == 0
        gate, up = want[:, 0::2], want[:, 1::2]
        silu = gate * torch.sigmoid(gate)
        _within(out, silu * up, 1.1 * up.abs() * slack[:, 0::2] + silu.abs() * slack[:, 1::2] + (silu * up).abs() * 2 ** -20)


@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 1200, 64), (4, 300, 128), (16, 300, 248),        # less than 256: the cut is added back
                                   (1, 1200, 256), (8, 300, 4096), (9, 2048, 4096),     # runs of four steps, loads of four, two and one ahead
                                   (16, 5200, 1032), (32, 5200, 4096), (32, 5200, 4104), (32, 130, 14336),   # 325 tiles: three CTAs to an SM
                                   (1, 1184, 4096), (2, 16, 520), (2, 1185, 4096),      # either side of the rule for few outputs
                                   (4, 592, 1024), (4, 593, 1024)])
def test_dense_matmul_of_few_rows_sums_like_fp32(M, N, K, positive):
    """fp32 results with the error of fp32 additions, not the tensor core's truncated ones.  A sum of K numbers by a tree or in short runs is off
    by up to three 2^-25 of itself (rms; signs at random, K 14336: the additions of 7 runs, of 4 steps and of a tree, each 2^-25 of its own
    result or less); a chain of truncated sums would be off by K / 512 * 2^-24 and more, always towards zero."""
    from proxy_inference_engine_b200 import _lib
    L = _lib.load_hybrid(build_if_missing=True)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    if positive:
        x, w = x.abs(), w.abs()
    want = x.double() @ w.double().t()
    out = torch.full((M, N), float("nan"), device="cuda")
    assert L.pieh_linear(_p(out), 1, N, _p(x), 0, K, _p(w), 0, None, M, N, K, 0, 0.0, None, None, 0, None) == 0
    off = out.double() - want
    assert off.norm() <= 3 * 2 ** -25 * want.norm(), float(off.norm() / want.norm())
    if positive and M * N >= 300:      # the mean of as many independent errors: no bias
        assert abs(float((off / want).mean())) <= 2 * 2 ** -25, float((off / want).mean())
    x[:, 3], w[0, 3] = float("inf"), 1.0      # an infinite product stays one
    assert L.pieh_linear(_p(out), 1, N, _p(x), 0, K, _p(w), 0, None, M, N, K, 0, 0.0, None, None, 0, None) == 0
    assert (out[:, 0] == float("inf")).all()


@pytest.mark.parametrize("W,shift", [(4, 0), (1028, 0), (4096, 0), (4096, 1), (1030, 0), (7, 0)])
def test_embedding_rows_by_four_and_by_one(W, shift):
    """Widths of whole fours, odd ones and a table that is not 16-byte aligned; the sums are of two values, so exact in fp32."""
    from proxy_inference_engine_b200 import _lib
    L, T, V, S = _lib.load_hybrid(), 3, 11, 2
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    tok, pos = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in ([10, 0, 4], [2, 0, 6]))
    for dt, code in ((torch.bfloat16, _lib.DTYPE_BF16), (torch.float32, _lib.DTYPE_F32)):
        table = torch.randn(V * W + 4, device="cuda").to(dt)[shift:shift + V * W].view(V, W)
        ptab = torch.randn(V, W, device="cuda").to(dt)
        xs = torch.empty(T, S, W, device="cuda")
        _lib.check_hybrid(L.pieh_embed_streams(_p(xs), _p(table), code, _p(tok), T, S, W, V, st), "embed_streams")
        assert torch.equal(xs, table[tok.long()].float()[:, None].expand(T, S, W))
        x, act = torch.empty(T, W, device="cuda"), torch.empty(T, W, device="cuda", dtype=torch.bfloat16)
        _lib.check_hybrid(L.pieh_embed_positions(_p(x), _p(act), _lib.DTYPE_BF16, _p(table), _p(ptab), code, _p(tok), _p(pos), T, W, V,
                                                 V, st), "embed_positions")
        want = table[tok.long()].float() + ptab[pos.long()].float()
        assert torch.equal(x, want) and torch.equal(act, want.to(torch.bfloat16))


@pytest.mark.parametrize("W", [4, 1020, 2052, 4096, 8192])
@pytest.mark.parametrize("rows", [148, 149])   # weights read ahead of the reductions, or behind them
def test_layer_norms_of_few_and_many_rows(rows, W):
    from proxy_inference_engine_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(W)
    x, y = (torch.randn(rows, W, generator=g, device="cuda") for _ in range(2))
    pw, pb, nw, nb = (torch.randn(W, generator=g, device="cuda") for _ in range(4))
    ln = lambda v, w, b: (v - v.mean(-1, keepdim=True)) / (v.var(-1, unbiased=False, keepdim=True) + 1e-5).sqrt() * w.double() + b.double()
    new = x.double() + ln(y.double(), pw, pb)
    want, h = ln(new, nw, nb), torch.empty(rows, W, device="cuda")
    _lib.check_hybrid(_lib.load_hybrid().pieh_layernorm_add(_p(x), _p(y), W, _p(pw), _p(pb), None, 0, None, _p(h), _lib.DTYPE_F32, _p(nw),
                                                            _p(nb), None, 1e-5, rows, W, C.c_void_p(torch.cuda.current_stream().cuda_stream)),
                      "layernorm_add")
    # sums in runs of at most 64 values and then pairwise; a row of 4 may be nearly constant, and its norm then enlarges the error
    # of the mean by 1 / sigma
    sd = new.std(-1, unbiased=False, keepdim=True) if W > 1 else 1.0
    size = new.abs().amax(-1, keepdim=True) * (1 + 1 / y.double().std(-1, unbiased=False, keepdim=True))
    _within(h, want, 2 ** -24 * 80 * (size / sd) * (1 + (want - nb.double()).abs() + nw.double().abs()) + 2 ** -23 * want.abs())


@pytest.mark.parametrize("H,G,dk,dv", [(16, 16, 128, 128), (8, 8, 16, 36), (8, 4, 32, 64)])
def test_delta_rule_of_one_portion_and_of_small_ones(H, G, dk, dv):
    """A portion prepared by warps and one scanned with registers to spare, against the same rows in small portions (prepared by CTAs)
    and single tokens (scanned with four CTAs on an SM).  The norms' sums are of other order: a few 2^-24 of a unit vector's size, and
    the recurrence, whose keys have length one, carries that on without enlarging it."""
    from proxy_inference_engine_b200 import _lib
    from proxy_inference_engine_b200.ragged import BatchDetails
    L = _lib.load_hybrid(build_if_missing=True)
    g = torch.Generator(device="cuda").manual_seed(dk)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    T, taps, nq = 400, 4, G * dk
    C_ = 2 * nq + H * dv
    ld = (C_ + H * dv + 2 * H + 3) // 4 * 4
    assert T * (2 * G + H) >= 6144 > 120 * (2 * G + H)      # either side of the rule between the two preparations
    conv_w, A, dt, norm, proj = rnd(C_, taps) * 0.3, rnd(H), rnd(H), torch.ones(dv, device="cuda"), rnd(T, ld)
    results = []
    for parts in ([T], [100, 120, 20, 110, 1, 1, 48]):
        conv, state = torch.zeros(1, taps - 1, C_, device="cuda"), torch.zeros(1, H, dk, dv, device="cuda")
        d = _lib.HybDelta(H, G, dk, dv, taps, conv_w.data_ptr(), A.data_ptr(), dt.data_ptr(), norm.data_ptr(), 1e-6, conv.data_ptr(),
                          state.data_ptr())
        outs, at = [], 0
        for n in parts:
            b = BatchDetails.build([("s", [1] * n, at, list(range(8)), 0)])
            desc, keep = b.hybrid_descriptor()
            q, k, v = (torch.full((n, w), float("nan"), device="cuda") for w in (nq, nq, H * dv))
            beta, decay, o = (torch.full((n, w), float("nan"), device="cuda") for w in (H, H, H * dv))
            rows = proj[at:at + n]
            assert L.pieh_delta_prepare(_p(q), _p(k), _p(v), _p(beta), _p(decay), _p(rows), ld, C.byref(d), C.byref(desc), None) == 0
            assert L.pieh_delta_scan(_p(o), _p(q), _p(k), _p(v), _p(beta), _p(decay), C.byref(d), C.byref(desc), None) == 0
            outs.append((q, k, v, beta, decay, o))
            at += n
        results.append([torch.cat(t) for t in zip(*outs)] + [conv, state])
        torch.cuda.synchronize()
    for name, a, b in zip(("q", "k", "v", "beta", "decay", "o", "conv", "state"), *results):
        assert torch.isfinite(a).all() and (a.double() - b.double()).norm() <= 1e-6 * b.double().norm(), name
