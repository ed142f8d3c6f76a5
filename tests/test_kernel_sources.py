"""Rules that every kernel's source keeps because breaking one could hang the GPU, so that no run may show it."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mini_llm_stack_b200" / "csrc"


def kernels(path):
    """(name, body) of the kernels of a source file, comments left out."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for m in re.finditer(r"__global__ void\b[^;{]*?(\w+_kernel)\(", text):
        body = text[m.end():]
        end = body.find("\n}\n")
        yield m.group(1), body[:end]


def with_tensor_memory():
    return [pytest.param(body, id=name) for path in sorted(CSRC.glob("*.cu")) for name, body in kernels(path)
            if "tmem_alloc" in body]


def test_the_kernels_are_found():
    assert len(with_tensor_memory()) == 10


@pytest.mark.parametrize("body", with_tensor_memory())
def test_successors_start_behind_the_allocation(body):
    """A kernel whose successor is resident while a block of its own still waits for tensor memory could wait for
    columns that the successor holds, and the successor for that kernel's end."""
    assert body.count("chain_release();") == 1
    assert re.search(r"if \(warp == \d\) \{\s*tmem_alloc(_pair)?\([^;]*;\s*chain_release\(\);\s*\}", body)
