"""pie_qmm_rows, several matrices and a residual in one launch of the prompt's matmul, against pie_qmm's tile kernel on each and pie_add, at every tile the choice
can take (pairs and single CTAs, K over a cluster's ranks) and at ragged widths.  One matrix, with or without a residual, which may be the output itself: the
same bits.  Several: the choice is the whole's, so that K may be cut in other places and fp32 sums added in another order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(g, n, k, bits):
    from proxy_inference_engine_b200 import nn
    lin = object.__new__(nn.QuantizedLinear)
    lin.group_size, lin.bits = 64, bits
    lin.weight = torch.randint(-(1 << 31), 1 << 31, (n, k * bits // 32), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    spread = 1 - 0.1 * torch.rand((n, k // 64), generator=g, device="cuda")
    lin.scales, lin.biases = (2 / k ** 0.5 / (2 ** bits - 1) * spread).bfloat16(), (-spread / k ** 0.5).bfloat16()
    return lin


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,K,widths", [(64, 4096, (256, 128, 128)), (70, 256, (200, 36, 7)), (129, 2048, (2048, 512, 512)), (300, 640, (264, 8)),
                                        (1000, 4096, (4096, 1024, 1024)), (1531, 2048, (2048, 512, 512)), (2100, 1024, (4000,)),
                                        (513, 512, (129, 129, 129))])
def test_one_launch_and_its_products_apart(monkeypatch, bits, M, K, widths):
    from proxy_inference_engine_b200 import nn, ops
    from proxy_inference_engine_b200._lib import QmvSeg, check, load
    monkeypatch.setenv("PIE_QMT", "0")                 # the separate calls on the tile kernel at 64 to 128 rows, too
    g = torch.Generator(device="cuda").manual_seed(M + K + bits)
    x, lins = torch.randn((M, K), generator=g, device="cuda").bfloat16(), tuple(_layer(g, n, K, bits) for n in widths)
    want = torch.cat([ops.quantized_matmul(x, l.weight, l.scales, l.biases, bits=bits) for l in lins], 1)
    n0 = load().pie_launch_count()
    got = nn.fused_prompt(x, lins)
    assert load().pie_launch_count() - n0 == 1
    # (other tile choices split K over other ranks, or not at all: sums of fp32 in another order, so that a value may fall on the other side)
    same = (got == want).float().mean()
    assert torch.isfinite(got).all() and same > 0.999 and (got.double() - want.double()).norm() <= 2 ** -12 * want.double().norm(), float(same)
    alone = nn.fused_prompt(x, lins[:1])
    assert torch.equal(alone, want[:, :widths[0]])     # the choice of a matrix alone: the same bits
    res = torch.randn((M, widths[0]), generator=g, device="cuda").bfloat16()
    want = ops.add(res, alone)
    assert torch.equal(nn.fused_prompt(x, lins[:1], residual=res), want)
    seg = (QmvSeg * 1)(QmvSeg(lins[0].weight.data_ptr(), lins[0].scales.data_ptr(), lins[0].biases.data_ptr(), widths[0]))
    check(load().pie_qmm_rows(res.data_ptr(), widths[0], x.data_ptr(), seg, 1, res.data_ptr(), M, K, 64, bits, torch.cuda.current_stream().cuda_stream), "in place")
    assert torch.equal(res, want)
