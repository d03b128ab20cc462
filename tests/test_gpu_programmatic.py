"""The switches for programmatic launches reach the matmuls as well: with them off a captured sequence has whole-kernel edges only."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


class _EdgeData(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]   # type 1: programmatic


def programmatic_edges(run):
    """(programmatic, all) edges of what run() launches, captured."""
    run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        run()
    rt, n = C.CDLL("libcudart.so.12"), C.c_size_t(256)
    src, dst, data = (C.c_void_p * 256)(), (C.c_void_p * 256)(), (_EdgeData * 256)()
    assert rt.cudaGraphGetEdges_v2(C.c_void_p(int(g.raw_cuda_graph())), src, dst, data, C.byref(n)) == 0
    return sum(data[i].type == 1 for i in range(n.value)), n.value


def _quantized(bits, rows):
    from proxy_inference_engine_b200 import nn, ops
    lin = nn.QuantizedLinear(1024, 1024, bias=False, bits=bits)
    x = torch.randn((rows, 1024), device="cuda").bfloat16()

    def run():
        y = x
        for _ in range(4):
            y = ops.quantized_matmul(y, lin.weight, lin.scales, lin.biases, bits=bits)
    return run


if __name__ == "__main__":
    for case in ((4, 200), (8, 200), (8, 16), (4, 100)):
        programmatic, edges = programmatic_edges(_quantized(*case))
        assert edges >= 3 and programmatic == 0, (case, programmatic, edges)


def test_quantized_matmuls():
    assert programmatic_edges(_quantized(4, 200))[0] >= 3


def test_quantized_matmuls_switched_off():
    run = subprocess.run([sys.executable, __file__], env={**os.environ, "PIE_PDL_AUX": "0", "PYTHONPATH": os.path.dirname(os.path.dirname(__file__))},
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]


def test_dense_matmuls():
    from proxy_inference_engine_b200 import _lib
    L = _lib.load_hybrid(build_if_missing=True)
    x, w, y = (torch.randn((512, 512), device="cuda").bfloat16() for _ in range(3))
    p = lambda t: C.c_void_p(t.data_ptr())

    def run():
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        for _ in range(4):
            assert L.pieh_linear(p(y), 0, 512, p(x), 0, 512, p(w), 0, None, 512, 512, 512, 0, 0.0, None, None, 0, stream) == 0

    try:
        got = []
        for on in (-1, 0, 1, -1):
            L.pieh_set_pdl(on)
            got.append(programmatic_edges(run))
    finally:
        L.pieh_set_pdl(-1)
    assert all(edges == 3 for _, edges in got) and [n for n, _ in got] == [3, 0, 3, 3]
