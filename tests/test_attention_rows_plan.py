"""Float32 attention: which steps' longer requests go by tiles (the bits are the same either way)."""

from types import SimpleNamespace

import pytest

from mini_llm_stack_b200.ops.kernels import Ops


@pytest.mark.parametrize("lens, before, heads, kv, span, tiles", [
    ([1, 1, 1], 4000, 32, 8, 0, False),              # decoded tokens
    ([8], 0, 32, 8, 0, False), ([32], 0, 32, 8, 0, True), ([8], 1024, 32, 8, 0, True),
    ([8] * 16, 0, 8, 8, 0, False),                   # four requests in a block, one after the other
    ([1] * 7 + [9], 1000, 8, 8, 0, False),           # decoded tokens would wait for the short portion
    ([1] * 31 + [512], 1000, 32, 8, 0, True),
    ([8], 8000, 32, 8, 4, False),                    # a window of four keys
])
def test_rule(lens, before, heads, kv, span, tiles):
    step = SimpleNamespace(ctx_lens=[before + n for n in lens], attn_tiles={})
    for _ in range(2):                               # worked out once a step
        assert Ops._rows_by_tiles(Ops, step, lens, heads, kv, span) is tiles
    assert len(step.attn_tiles) == (1 if max(lens) >= 8 else 0)


def test_unknown_contexts_go_by_tiles():
    assert Ops._rows_by_tiles(Ops, SimpleNamespace(), [8, 1], 32, 8, 0)
    assert not Ops._rows_by_tiles(Ops, SimpleNamespace(), [7, 1], 32, 8, 0)
