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


def roles(body):
    """The parts of a kernel that its warps take by their number."""
    return re.split(r"(?=\n +(?:if \(warp |\} else if \(warp |\} else \{\n))", body)


def waiting_roles():
    return [pytest.param(role, id=f"{name}-{i}") for path in sorted(CSRC.glob("*.cu")) for name, body in kernels(path)
            if "tmem_alloc" in body for i, role in enumerate(roles(body)) if re.search(r"mbar_wait\w*\(", role)]


@pytest.mark.parametrize("role", waiting_roles())
def test_lanes_leave_a_loop_together(role):
    """Where a wait that runs out takes a warp out of a loop, all of its lanes go: those that stayed would wait for
    the others at the next instruction that a whole warp executes."""
    together = re.search(r"elect_one|tmem_ld|tmem_st|_sync\(0xffffffffu|__syncwarp", role)
    leaves = re.search(r"\bbreak;|return false;|&& !timed_out;", role)
    one_lane = "lane == 0) {\n" in role[:250]
    if together and leaves and not one_lane:
        assert not re.search(r"mbar_wait(_cluster)?\(", role), "a wait that each lane judges by itself"


@pytest.mark.parametrize("body", [p for p in with_tensor_memory() if "tma_load_2d" in p.values[0] or "bulk_load" in p.values[0]])
def test_copies_land_before_the_block_ends(body):
    """The role that copies waits, behind its last copy, until those under way are there: also where a wait ran out."""
    parts = re.split(r"\n    (?:if|\} else if) \(warp ", body)
    role = next(r for r in parts if "tma_load_2d" in r or "load_k(c + 2)" in r)
    behind = role[max(m.end() for m in re.finditer(r"tma_load_2d\w*\(|load_[kqtp]\(c", role)):]
    assert re.search(r"for \(int \w+ = [^;]*;[^)]*\)\s*if \(!mbar_wait\w*\([^;]*(full|FULL)[^;]*timed_out = true;", behind)


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.stem)
def test_shared_memory_limits_never_fall(path):
    """A launcher that remembers what limit it set a kernel sets one and the same each time: with a limit for every
    launch, two threads could leave the lower one behind and the memory of the higher."""
    assert not re.search(r"static int \w*configured", path.read_text())
