"""Kernels that allocate tensor memory let their dependents start behind that: a dependent takes its own ahead of its wait, and what it holds while it waits for a
grid that is waiting for tensor memory is held for good."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "proxy_inference_engine_b200" / "csrc"


def _kernels():
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for part in re.split(r"__global__", text)[1:]:
            body = part.split("\n}\n")[0]
            if "tcgen05.alloc" in body:
                yield pytest.param(body, id=f"{path.name}:{re.search(r'(\w+)\s*\(const', body).group(1)}")


@pytest.mark.parametrize("body", list(_kernels()))
def test_tensor_memory_comes_before_the_dependents(body):
    alloc = body.rindex("tcgen05.alloc")
    assert all(m.start() > alloc for m in re.finditer(r"pdl_launch_dependents\(\)|pdl_sync\(\)|griddepcontrol\.launch_dependents", body))


def test_there_are_such_kernels():
    assert len(list(_kernels())) >= 6
