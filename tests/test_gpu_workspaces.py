"""Split decode attention and the matmuls on several streams, threads and graphs at a time: every call adds up its own partial results."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(seed):
    from proxy_inference_engine_b200 import ops
    from proxy_inference_engine_b200.cache import QuantizedKVCache
    g = torch.Generator(device="cuda").manual_seed(seed)
    cache = QuantizedKVCache(64, 8, 4000)
    cache.update_and_fetch(*(torch.randn((2, 8, 4000, 128), generator=g, device="cuda").bfloat16() for _ in "kv"))
    q, pos = torch.randn((2, 32, 128), generator=g, device="cuda").bfloat16(), torch.full((2,), 3999, dtype=torch.int32, device="cuda")
    return lambda: ops.decode_attention_q8(q, cache.desc(), pos, 128 ** -0.5, 8, max_context=4000)


def test_two_streams():
    calls = [_case(i) for i in range(2)]
    want = [f() for f in calls]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in calls], [[], []]
    for _ in range(50):
        for f, s, out in zip(calls, streams, got):
            with torch.cuda.stream(s):
                out.append(f())
    torch.cuda.synchronize()
    assert all(torch.equal(y, w) for out, w in zip(got, want) for y in out)


def test_two_threads():
    calls, got = [_case(i) for i in range(2)], [[], []]
    want = [f() for f in calls]
    torch.cuda.synchronize()

    def run(f, out):
        with torch.cuda.stream(torch.cuda.Stream()):
            out.extend(f() for _ in range(50))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=run, args=a) for a in zip(calls, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [len(out) for out in got] == [50, 50]
    assert all(torch.equal(y, w) for out, w in zip(got, want) for y in out)


def test_a_graph_beside_eager_calls():
    """A geometry first met in a capture, an eager call of it before any replay, a larger one that replaces the eager call's buffer, then replays."""
    from proxy_inference_engine_b200 import ops
    f, larger = _case(3), _case(4)
    f()                                         # (kernels opt in to their shared memory ahead of the capture)
    ops.workspaces.mine.eager.clear()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = f()
        again = f()
    want = f()
    for key in list(ops.workspaces.mine.eager):
        ops.workspaces.get(key[0], 1 << 24, torch.device("cuda", key[1]))
    other = larger()
    for _ in range(3):
        out.zero_()
        again.zero_()
        graph.replay()
        assert torch.equal(out, want) and torch.equal(again, want)
    assert torch.equal(larger(), other) and torch.equal(f(), want)
