"""GPU parity on the benchmark's own configurations (not a toy model), against the CPU oracle (mode B = fp32
inside every MLX op, bf16 at the op boundaries: what MLX computes for a bf16 checkpoint).

Correct means: per-layer bf16 activations within 2e-2 relative error and identical greedy tokens
over 128 steps.  On random-init weights the logits over 128 256 classes are nearly flat, so a greedy token can flip on a
near-tie from fp32 summation order alone: tokens are compared teacher-forced, a mismatch only counts when
the oracle's own gap between the two candidates exceeds twice the largest logit difference seen on that step, and the
exact-match run length (= how far a free-running decode stays identical) is reported.
Reference loop: PIE/engine/inference_engine.py:228-297 -> PIE/models/llama/language.py:199-210."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from parity_util import make_oracle, n2t_bf16, n2t_words, rel_l2, run_decode_parity, t2n

pytestmark = pytest.mark.gpu
TOL = 2e-2
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def greedy_parity(args, prompt_len, steps, seed=0, max_context=None, engine_kw=None):
    """Prefill + `steps` teacher-forced greedy steps of DecodeEngine against LlamaOracle.  Returns a report."""
    from proxy_inference_engine_b200.checkpoint import build_model, random_weights
    from proxy_inference_engine_b200.decode import DecodeEngine

    w = random_weights(args, seed=seed, device="cuda", gen_device="cpu")
    model = build_model(args, w)
    o = make_oracle(args, w)
    prompt = torch.randint(0, args.vocab_size, (1, prompt_len), generator=torch.Generator().manual_seed(1))
    eng = DecodeEngine(model, batch=1, max_context=max_context or prompt_len + steps + 2, **(engine_kw or {}))
    eng.prefill(prompt)
    caches, trace = o.make_cache(), {}
    lo = o(prompt.numpy(), caches, trace=trace)[:, -1]
    # per-layer activations of the prompt: every layer's K and V rows are functions of that layer's input stream
    kv_err = []
    for i, c in enumerate(eng.cache):
        kv_err.append(max(rel_l2(c.keys[:, :, :prompt_len].float().cpu().numpy(), caches[i].keys[:, :, :prompt_len]),
                          rel_l2(c.values[:, :, :prompt_len].float().cpu().numpy(), caches[i].values[:, :, :prompt_len])))
    errs, flips, strong, first_flip = [], 0, 0, None
    for s in range(steps):
        lg = eng.logits.float().cpu().numpy()
        errs.append(rel_l2(lg, lo))
        tok_o, tok_g = int(lo[0].argmax()), int(eng.tokens[0].item())
        if tok_o != tok_g:
            flips += 1
            if first_flip is None:
                first_flip = s
            gap = float(lo[0, tok_o] - lo[0, tok_g])
            if gap > 2.0 * float(np.abs(lg - lo).max()):
                strong += 1
        eng.tokens.copy_(torch.tensor([tok_o], dtype=torch.int32))  # teacher forcing
        eng.step(1)
        lo = o(np.array([[tok_o]], np.int32), caches)[:, -1]
    return {"steps": steps, "max_logit_rel_err": max(errs), "max_kv_rel_err": max(kv_err), "near_tie_flips": flips,
            "strong_mismatch": strong, "exact_match_run": steps if first_flip is None else first_flip}


def test_config1_llama_3_2_1b_q4_128_prompt_128_greedy_steps():
    """Llama-3.2-1B random-init, MLX q4 gs64, bs1, 128-token prompt + 128 greedy steps."""
    from proxy_inference_engine_b200.checkpoint import preset_args
    args = preset_args("llama-3.2-1b", bits=4)
    rep = greedy_parity(args, prompt_len=128, steps=128)
    print("config1 parity:", rep)
    assert rep["max_kv_rel_err"] < TOL, rep        # per-layer activations (all 16 layers' K/V of the prompt)
    assert rep["max_logit_rel_err"] < TOL, rep     # every step's logits
    assert rep["strong_mismatch"] == 0, rep        # greedy tokens identical wherever the oracle's choice is not a near-tie
    assert rep["exact_match_run"] >= 16, rep


@pytest.mark.parametrize("bits,paged", [(4, False), (4, True), (8, False), (8, True)])
def test_one_8b_shaped_layer_decodes_like_the_oracle(bits, paged):
    """One transformer layer with Llama-3.1-8B's shapes (h 4096, ffn 14336, 32/8 heads, D 128; vocabulary cut to 4096)
    through the CUDA-graph engine: the kernels run on the 8B matrices' real dimensions (configs 2 and 3)."""
    from proxy_inference_engine_b200.checkpoint import preset_args
    args = preset_args("llama-3.1-8b", bits=bits, num_hidden_layers=1, vocab_size=4096)
    rep = run_decode_parity(args, prompt_len=40, steps=16, batch=2 if paged else 1, paged=paged)
    assert rep["max_rel_err"] < TOL, rep
    assert rep["strong_mismatch"] == 0, rep


@pytest.mark.parametrize("N,K", [(28672, 4096), (128256, 4096)])
def test_batched_decode_default_routing_at_8b_q8_shapes(N, K):
    """Config 3's GEMMs (8B q8, 32 rows) on the library's DEFAULT routing (tcgen05 kernel where it pays)."""
    from oracle import oracle as orc
    from proxy_inference_engine_b200 import ops
    rng = np.random.default_rng(N)
    w = (rng.uniform(-1, 1, (N, K)) / np.sqrt(K)).astype(np.float32)
    wq, s, b = orc.quantize(w, 64, 8)
    x = orc.round_bf16(rng.standard_normal((32, K)).astype(np.float32))
    ref = orc.quantized_matmul(x, wq, s, b, True, 64, 8, mode="B")
    got = t2n(ops.quantized_matmul(n2t_bf16(x), n2t_words(wq), n2t_bf16(s), n2t_bf16(b), True, 64, 8))
    # the tcgen05 form rounds the dequantized weight to bf16 before the MMA (the rounding structure of Metal qmm_t,
    # kernels/quantized.h:411-417): judged by relative L2 like tests/test_gpu_attn_fused.py, plus a loose per-element bound
    assert rel_l2(got, ref) < 3e-3
    assert np.all(np.abs(got - ref) <= np.abs(ref) * 2.0 ** -5 + 1e-2 * np.abs(ref).max())


def test_decode_attention_simt_form(monkeypatch):
    """The SIMT split-K decode attention (PIE_DECODE_ATTN=simt, read once per process: run in a child)."""
    code = (
        "import numpy as np, torch, sys; sys.path.insert(0, %r); sys.path.insert(0, %r)\n"
        "from oracle import oracle as orc\n"
        "from proxy_inference_engine_b200 import ops\n"
        "from parity_util import n2t_bf16, t2n, rel_l2\n"
        "rng = np.random.default_rng(0)\n"
        "for (B, Hq, Hkv, D, T) in ((1, 8, 2, 128, 300), (3, 4, 4, 64, 77), (2, 16, 2, 128, 1100)):\n"
        "    q = orc.round_bf16(rng.standard_normal((B, Hq, 1, D)).astype(np.float32))\n"
        "    k = orc.round_bf16(rng.standard_normal((B, Hkv, T, D)).astype(np.float32))\n"
        "    v = orc.round_bf16(rng.standard_normal((B, Hkv, T, D)).astype(np.float32))\n"
        "    ref = orc.scaled_dot_product_attention(q, k, v, D ** -0.5, None, -1, 'B')\n"
        "    got = t2n(ops.scaled_dot_product_attention(n2t_bf16(q), n2t_bf16(k), n2t_bf16(v), scale=D ** -0.5))\n"
        "    assert rel_l2(got, ref) < 1e-2, rel_l2(got, ref)\n"
        "print('SIMT_OK')\n") % (ROOT, os.path.join(ROOT, "tests"))
    env = dict(os.environ, PIE_DECODE_ATTN="simt")
    out = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "SIMT_OK" in out.stdout, out.stdout + out.stderr


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="tensor-parallel parity needs two GPUs")
def test_tensor_parallel_two_gpus_matches_single_gpu():
    """tools/tp_check.py under torchrun: the sharded engine against the single-GPU engine (tokens + logits)."""
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node", "2", "--master-addr",
           "127.0.0.1", "--master-port", "29533", os.path.join(ROOT, "tools", "tp_check.py")]
    for fused in ("0", "1"):   # the stand-alone one-shot exchange kernels, then the exchange fused into the GEMVs (bs1)
        out = subprocess.run(cmd, capture_output=True, text=True, timeout=900, env=dict(os.environ, PIE_TP_FUSED=fused))
        assert out.returncode == 0 and "TP_CHECK PASS" in out.stdout, out.stdout[-2000:] + out.stderr[-2000:]
        assert ("_fused" in out.stdout) == (fused == "1")
