"""pie_qmt (csrc/pie_qmt.cuh), some dozens of rows with the weights through tensor memory, against float64 at the edges of its rows, tiles and
shares.  Weights are exact, activations are down to 2^-25 (8 bits: 2^-21) of a row's largest, and sums are off by less than 1e-6, so what is left is the
rounding of the result to bf16: 2^-9 of a value at the most, in the 2-norm 2^-9 / sqrt(3) = 1.13e-3 to 1.95e-3 as the values lie in their binade.  Two tests
below look under that: products next to zero show the sums, a large value that meets no weight the activations."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(g, n, k, bits):
    words = torch.randint(-(1 << 31), 1 << 31, (n, k * bits // 32), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    spread = 1 - 0.1 * torch.rand((n, k // 64), generator=g, device="cuda")
    return [words, (2 / k ** 0.5 / (2 ** bits - 1) * spread).bfloat16(), (-spread / k ** 0.5).bfloat16()]


def _dense(m, bits):
    words, s, b = m
    q = ((words[:, :, None] >> torch.arange(0, 32, bits, device="cuda", dtype=torch.int32)) & (2 ** bits - 1)).reshape(s.shape + (64,)).double()
    return (q * s.double()[:, :, None] + b.double()[:, :, None]).flatten(1)


def _call(x, mats, bits, norm=None, residual=None, swiglu=False):
    from proxy_inference_engine_b200 import _lib
    L = _lib.load()
    segs = (_lib.QmvSeg * len(mats))()
    for seg, (w, s, b) in zip(segs, mats):
        seg.wq, seg.scales, seg.biases, seg.N = w.data_ptr(), s.data_ptr(), b.data_ptr(), w.shape[0]
    M, K = x.shape
    N = sum(m[0].shape[0] for m in mats) // (2 if swiglu else 1)
    nb = L.pie_qmt_scratch_bytes(M, N, K, 64, bits, int(swiglu))
    scratch = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")            # its contents do not matter
    out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    p = lambda t: None if t is None else t.data_ptr()
    n0 = L.pie_launch_count()
    _lib.check(L.pie_qmt(p(out), N, p(x), K, M, K, segs, len(mats), 64, bits, p(norm), 1e-5, 2 if swiglu else 0 if residual is None else 1,
                         p(residual), p(scratch), nb, torch.cuda.current_stream().cuda_stream), "qmt")
    assert L.pie_launch_count() - n0 == 2 and L.pie_pipeline_error() == 0
    return out


def _rel(y, ref):
    return float((y.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,N,K", [(1, 128, 512), (16, 129, 1536), (17, 2048, 2048), (32, 19200, 512), (33, 300, 8192), (48, 1000, 28672),
                                   (49, 4096, 4096), (64, 6144, 512), (80, 257, 4608), (97, 512, 512), (128, 22000, 1024)])
def test_products_match_float64(bits, M, N, K, monkeypatch):
    monkeypatch.setenv("PIE_QMT", "2")
    g = torch.Generator(device="cuda").manual_seed(M + N + K + bits)
    m, x = _matrix(g, N, K, bits), torch.randn((M, K), generator=g, device="cuda").bfloat16()
    if M > 3:
        x[1] *= 1e-30
        x[2, : K // 2] *= 2.0 ** -12          # half of a row far below its largest values
        x[3] = 0
    y, ref = _call(x, [m], bits), x.double() @ _dense(m, bits).t()
    assert _rel(y, ref) < 2e-3
    for r in {0, 1, 2, M - 1} & set(range(M)):
        assert _rel(y[r], ref[r]) < 2.5e-3
    assert M <= 3 or not y[3].any()


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M", [23, 70])
def test_norm_segments_residual_and_swiglu(bits, M, monkeypatch):
    from proxy_inference_engine_b200 import ops
    monkeypatch.setenv("PIE_QMT", "2")
    K = 2048
    g = torch.Generator(device="cuda").manual_seed(M + bits)
    x, nw = (3 * torch.randn((M, K), generator=g, device="cuda")).bfloat16(), (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).bfloat16()
    mats = [_matrix(g, n, K, bits) for n in (520, 128, 130)]
    xn = ops.rms_norm(x, nw, 1e-5).double()
    # (the norm's sum of squares has another order: a normalised value may fall on the other side of a rounding boundary)
    assert _rel(_call(x, mats, bits, norm=nw), torch.cat([xn @ _dense(m, bits).t() for m in mats], 1)) < 2.2e-3
    res = torch.randn((M, 520), generator=g, device="cuda").bfloat16()
    assert _rel(_call(x, mats[:1], bits, residual=res), res.double() + x.double() @ _dense(mats[0], bits).t()) < 2.6e-3    # two roundings
    gate, up = _matrix(g, 9500, K, bits), _matrix(g, 9500, K, bits)
    a, b = x.double() @ _dense(gate, bits).t(), x.double() @ _dense(up, bits).t()
    assert _rel(_call(x, [gate, up], bits, swiglu=True), torch.nn.functional.silu(a) * b) < 4.5e-3                           # five roundings


@pytest.mark.parametrize("bits", [4, 8])
def test_scales_no_operand_holds_and_values_that_are_no_numbers(bits, monkeypatch):
    monkeypatch.setenv("PIE_QMT", "2")
    M, N, K = 19, 300, 4096
    g = torch.Generator(device="cuda").manual_seed(bits)
    m, x = _matrix(g, N, K, bits), torch.randn((M, K), generator=g, device="cuda").bfloat16()
    w, s, b = m
    s[5, 3], s[77, 0], b[200, 10], b[131] = 1e-12, 50.0, 1e5, 1e-9
    s[130] *= 1e20
    b[130] *= 1e20
    s[299], b[299] = 0, 0
    s[140], b[140] = 1e-7, 0                                     # what a group of zeros quantizes to
    y, ref = _call(x, [m], bits), x.double() @ _dense(m, bits).t()
    for n in list(range(0, 299, 13)) + [5, 77, 130, 131, 140, 200]:
        assert _rel(y[:, n], ref[:, n]) < 4e-3, n
    assert not y[:, 299].any()
    x[2, 5], x[7, 9] = float("inf"), float("nan")
    z = _call(x, [m], bits)
    keep = [r for r in range(M) if r not in (2, 7)]
    assert torch.equal(z[keep], y[keep]) and z[7].isnan().all() and not z[2].isfinite().any()


def test_few_rows_share_their_bits_with_any_batch(monkeypatch):
    """A row's result does not depend on the rows beside it, nor a call's on the one before it."""
    monkeypatch.setenv("PIE_QMT", "2")
    g = torch.Generator(device="cuda").manual_seed(3)
    m, x = _matrix(g, 4096, 4096, 4), torch.randn((32, 4096), generator=g, device="cuda").bfloat16()
    y = _call(x, [m], 4)
    assert torch.equal(_call(x[:20].contiguous(), [m], 4), y[:20]) and torch.equal(_call(x, [m], 4), y)


@pytest.mark.parametrize("bits", [4, 8])
def test_the_native_host_form_is_the_python_one(bits, monkeypatch):
    """csrc/pie_host.cpp against nn.fused_rows without it: the same bits where it answers, and no answer where that has none."""
    from proxy_inference_engine_b200 import nn, ops
    assert ops.native_fused_rows().__name__ == "fused_rows"
    g = torch.Generator(device="cuda").manual_seed(bits)
    K = 2048

    def layer(n):
        lin = object.__new__(nn.QuantizedLinear)
        lin.group_size, lin.bits = 64, bits
        lin.weight, lin.scales, lin.biases = _matrix(g, n, K, bits)
        return lin

    lins, norm = (layer(6144), layer(6144)), object.__new__(nn.RMSNorm)
    norm.weight, norm.eps = torch.ones(K, dtype=torch.bfloat16, device="cuda"), 1e-5
    native = lambda x, ls=lins, n=None, r=None, s=False: ops.native_fused_rows()(x, ls, n, r, s, nn.QuantizedLinear, nn.RMSNorm, ops.qmv_workspace)
    for shape in ((1, K), (2, 1, K), (20, K), (3, 13, K), (100, K), (0, K)):
        x = torch.randn(shape, generator=g, device="cuda").bfloat16()
        for kw in (dict(), dict(norm=norm), dict(swiglu=True), dict(residual=torch.randn(shape[:-1] + (6144,), generator=g, device="cuda").bfloat16())):
            ls = lins if "residual" not in kw else lins[:1]
            mine = native(x, ls, kw.get("norm"), kw.get("residual"), kw.get("swiglu", False))
            with monkeypatch.context() as m:
                m.setattr(ops, "native_fused_rows", lambda: lambda *a: None)
                want = nn.fused_rows(x, ls, **kw)
            assert (mine is None) == (want is None) and (mine is None or (mine.shape == want.shape and torch.equal(mine, want)))
    x = torch.randn((4, K), generator=g, device="cuda").bfloat16()
    biased, other, strided, wide = layer(256), layer(256), layer(256), layer(256)
    biased.bias = torch.zeros(256, device="cuda")
    other.group_size = 32
    strided.scales = strided.scales.t().contiguous().t()
    wide.scales = wide.scales.float()
    for bad in (biased, other, strided, wide, lambda v: v):
        assert native(x, (bad,)) is None
    assert native(x.float()) is None and native(x[:, ::2]) is None and native(x.t()) is None and native(x[:, :1024].contiguous()) is None
    assert native(x, lins[:1], None, x) is None and native(x, lins, lambda v: v) is None and native(x, list(lins)) is None
    assert torch.func.vmap(lambda v: torch.zeros(()) if native(v) is None else torch.ones(()))(x[:, None]).sum() == 0


def _near_zero_targets(g, M, K, w):
    """x [M, K] whose product with row m of w is far below the sums it is made of: what comes out is the sums' own error, which no rounding of
    the result hides.  Projected off w's row first, then corrected in one small element after the other."""
    x, rows = torch.randn((M, K), generator=g, device="cuda"), w[:M]
    x = (x.double() - (x.double() * rows).sum(1, keepdim=True) / (rows * rows).sum(1, keepdim=True) * rows).bfloat16()
    at = torch.arange(M, device="cuda")
    for _ in range(6):
        r = (x.double() * rows).sum(1)
        k = torch.where(rows.abs() >= rows.abs().median(), x.double().abs(), torch.inf).argmin(1)
        x[at, k] = (x[at, k].double() - r / rows[at, k]).bfloat16()
    return x


@pytest.mark.parametrize("bits,M,K", [(4, 9, 512), (4, 16, 4096), (4, 32, 1536), (4, 32, 14336), (4, 48, 14336), (4, 63, 4608), (8, 20, 4096), (8, 48, 8192)])
def test_sums_are_no_further_off_than_the_gemvs(bits, M, K, monkeypatch):
    """Before their rounding to bf16, over a tile's whole K in one CTA (as many tiles as SMs).  The tensor core cuts the sums it returns, towards zero: with
    one accumulator for all of K they were off by 1.8e-6 of a product's size at K 4096 and 8.0e-6 at 14336, the GEMV by 1.1e-6 to 1.4e-6 at every K."""
    from proxy_inference_engine_b200 import _lib
    L, N = _lib.load(), 128 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(M + K + bits)
    m = _matrix(g, N, K, bits)
    w = _dense([t[:128] for t in m], bits)
    size = float((torch.randn((64, K), generator=g, device="cuda").double() @ w.t()).norm() / (64 * 128) ** 0.5)      # of a product of N(0, 1) rows
    mine, theirs = [], []
    for _ in range(3):
        x = _near_zero_targets(g, M, K, w)
        ref = (x.double() * w[:M]).sum(1)
        assert ref.abs().max() < 2e-5 * size                              # its rounding to bf16: at most 4e-8 of a product's size
        monkeypatch.setenv("PIE_QMT", "2")
        mine.append(_call(x, [m], bits).diagonal().double() - ref)
        monkeypatch.setenv("PIE_QMT", "0")
        y, nb = torch.empty((M, N), dtype=torch.bfloat16, device="cuda"), L.pie_qmv_workspace_bytes(M, N, K, bits, 0, 0)
        ws = torch.zeros(max(nb, 256), dtype=torch.uint8, device="cuda")
        _lib.check(L.pie_qmv(y.data_ptr(), x.data_ptr(), *(t.data_ptr() for t in m), M, N, K, 64, bits, ws.data_ptr(), ws.numel(),
                             torch.cuda.current_stream().cuda_stream), "qmv")
        theirs.append(y.diagonal().double() - ref)
    off = [float(torch.cat(v).square().mean().sqrt()) / size for v in (mine, theirs)]
    assert off[0] <= off[1] and off[0] < 1e-6, off


def test_a_call_holds_the_weights_it_was_made_with():
    """Another thread may put other tensors in a layer's place while a call looks for its workspace: the memory of those the call has read about must
    not be given to anybody before its launch is queued."""
    from proxy_inference_engine_b200 import nn, ops
    g = torch.Generator(device="cuda").manual_seed(5)
    lin, norm, x = object.__new__(nn.QuantizedLinear), object.__new__(nn.RMSNorm), torch.randn((20, 2048), generator=g, device="cuda").bfloat16()
    lin.group_size, lin.bits = 64, 4
    norm.eps = 1e-5

    def call(workspace):
        torch.cuda.synchronize()
        lin.weight, lin.scales, lin.biases = _matrix(torch.Generator(device="cuda").manual_seed(6), 512, 2048, 4)
        norm.weight = torch.ones(2048, dtype=torch.bfloat16, device="cuda")
        return ops.native_fused_rows()(x, (lin,), norm, None, False, nn.QuantizedLinear, nn.RMSNorm, workspace)

    others, asked = [], []

    def swap(nbytes, device):
        asked.append(nbytes)
        for owner, name in ((lin, "weight"), (lin, "scales"), (lin, "biases"), (norm, "weight")):
            shape, dtype = getattr(owner, name).shape, getattr(owner, name).dtype
            setattr(owner, name, None)
            others.append(torch.ones(shape, dtype=dtype, device="cuda"))      # the allocator's next block of this size: the one given back, if any was
        return ops.qmv_workspace(nbytes, device)

    want, got = call(ops.qmv_workspace), call(swap)
    assert asked and torch.equal(got, want)


@pytest.mark.parametrize("bits,M,K,top", [(4, 4, 14336, 23), (4, 16, 4096, 23), (4, 63, 1536, 23), (8, 40, 4096, 19)])
def test_small_values_beside_a_large_one(bits, M, K, top, monkeypatch):
    """2^top in a group of zero weights, in rows of N(0, 1): the others are what fp16 leaves them under the row's power of two, off by at most 2^-33 (8 bits:
    2^-29) of the largest value, which makes 2^-10 / sqrt(3) = 5.6e-4 of a product, below the 1.95e-3 of its rounding: 2.03e-3 together."""
    monkeypatch.setenv("PIE_QMT", "2")
    g = torch.Generator(device="cuda").manual_seed(M + K)
    m, x = _matrix(g, 256, K, bits), torch.randn((M, K), generator=g, device="cuda").bfloat16()
    m[1][:, 0], m[2][:, 0] = 0, 0
    x[:, 15] = 2.0 ** top
    assert _rel(_call(x, [m], bits), x.double() @ _dense(m, bits).t()) < 2.1e-3


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,K", [(16, 512), (40, 4096), (64, 4096), (77, 14336), (128, 28672)])
def test_rows_with_infinities(bits, M, K, monkeypatch):
    """Infinities of one sign or of both, first and last of a row, against float64: an infinity times the weights' signs, NaN where they disagree or a weight
    is zero; marked rows of the matrix among them, and the rows beside as they are without."""
    monkeypatch.setenv("PIE_QMT", "2")
    g = torch.Generator(device="cuda").manual_seed(M + K + bits)
    m, x = _matrix(g, 200, K, bits), torch.randn((M, K), generator=g, device="cuda").bfloat16()
    m[1][5, 0], m[2][9, 0] = 50.0, 1e5                                  # marked
    m[1][:, 3], m[2][:, 3] = 0, 0                                       # weights of zero at k 192 .. 255
    inf = float("inf")
    y = _call(x, [m], bits)
    x[0, 0], x[1, K - 1], x[2, 7], x[2, K // 2], x[3, 200], x[M - 1, :] = inf, -inf, inf, -inf, inf, inf
    x[4, 11], x[4, 12] = inf, float("nan")
    z, ref = _call(x, [m], bits).double(), x.double() @ _dense(m, bits).t()
    hit = [0, 1, 2, 3, 4, M - 1]
    assert torch.equal(z[hit].nan_to_num(0.0), ref[hit].nan_to_num(0.0)) and torch.equal(z[hit].isnan(), ref[hit].isnan())
    assert z[0].isinf().all() and z[2].isnan().any() and z[2].isinf().any() and z[3].isnan().all()
    rest = [r for r in range(M) if r not in hit]
    assert torch.equal(z[rest], y[rest].double())


def test_a_decode_engine_has_room_for_it_at_more_than_32_rows(monkeypatch):
    """The workspace of a step of 40 rows holds what the tensor-memory matmul asks for with 40 rows, or the step would fall back to passes of 32; and the
    captured step's logits are those of the kernels without it."""
    from parity_util import tiny_args
    from proxy_inference_engine_b200 import _lib
    from proxy_inference_engine_b200.decode import DecodeEngine
    from proxy_inference_engine_b200.llama import Model
    B, L = 40, _lib.load()
    model = Model(tiny_args(hidden_size=2048, intermediate_size=2048, num_hidden_layers=1, num_attention_heads=32, num_key_value_heads=8))
    eng, ids = DecodeEngine(model, B, 64), torch.randint(0, 640, (B, 6), device="cuda")
    for n, k, dual in ((3072, 2048, 0), (2048, 2048, 0), (2048, 2048, 1)):
        need = L.pie_qmt_scratch_bytes(B, n, k, 64, 4, dual)
        assert need and eng.qmv_ws.numel() >= (128 << 10) + need
    eng.prefill(ids)
    first = eng.tokens.clone()
    eng.step(1)
    logits = eng.logits.double().clone()
    monkeypatch.setenv("PIE_QMT", "0")
    other = DecodeEngine(model, B, 64)
    other.prefill(ids)
    other.tokens.copy_(first)
    other.step(1)
    assert _rel(logits, other.logits.double()) < 2e-2


def _many_rows(g, K=2048, n=6144, rows=48):
    from proxy_inference_engine_b200 import nn
    lin = object.__new__(nn.QuantizedLinear)
    lin.group_size, lin.bits = 64, 4
    lin.weight, lin.scales, lin.biases = _matrix(g, n, K, 4)
    return lin, torch.randn((rows, K), generator=g, device="cuda").bfloat16()


def _native(x, lin):
    from proxy_inference_engine_b200 import nn, ops
    y = ops.native_fused_rows()(x, (lin,), None, None, False, nn.QuantizedLinear, nn.RMSNorm, ops.qmv_workspace)
    assert y is not None
    return y


def test_the_native_form_on_a_stream_of_its_own_and_in_a_capture():
    lin, x = _many_rows(torch.Generator(device="cuda").manual_seed(8))
    want, twice = _native(x, lin), _native(2 * x, lin)
    side, a = torch.cuda.Stream(), torch.randn((8192, 8192), device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        late = x * 0
        for _ in range(3):
            torch.mm(a, a)                                               # the copy below comes behind it, and the call behind that
        late.copy_(x)
        got = _native(late, lin)
    side.synchronize()
    assert torch.equal(got, want)
    graph, fed = torch.cuda.CUDAGraph(), x.clone()
    with torch.cuda.graph(graph):
        out = _native(fed, lin)
    for v, y in ((x, want), (2 * x, twice), (x, want)):
        fed.copy_(v)
        graph.replay()
        assert torch.equal(out, y)


def test_two_threads_call_the_native_form_on_streams_of_their_own():
    from concurrent.futures import ThreadPoolExecutor
    g = torch.Generator(device="cuda").manual_seed(9)
    work = [_many_rows(g), _many_rows(g, n=4000, rows=63)]
    want = [_native(x, lin) for lin, x in work]
    torch.cuda.synchronize()

    def loop(i):
        (lin, x), bad = work[i], 0
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(200):
                bad += int(not torch.equal(_native(x, lin), want[i]))
        return bad

    with ThreadPoolExecutor(2) as pool:
        assert list(pool.map(loop, range(2))) == [0, 0]
