"""Chunk-wise scans: how a step's chunks are cut into parts that fit scratch."""

import random

from mini_llm_stack_b200.ops.kernels import Ops


def test_parts_cover_every_chunk_once_in_order():
    rng = random.Random(1)
    for _ in range(500):
        each = [rng.randint(1, 40) for _ in range(rng.randint(1, 30))]
        most = rng.randint(1, 60)
        done = [0] * len(each)
        for at, n, first, span, total in Ops._chunk_parts(each, most):
            counts = [min(max(c - first, 0), span) for c in each[at:at + n]]
            assert sum(counts) == total <= most and min(counts) >= 1
            for i, c in enumerate(counts):
                assert done[at + i] == first          # a request's chunks go on where the part before ended
                done[at + i] += c
        assert done == each


def test_whole_requests_stay_together():
    assert Ops._chunk_parts([5, 70, 1, 1, 64], 64) == [
        (0, 1, 0, 5, 5), (1, 1, 0, 64, 64), (1, 1, 64, 6, 6), (2, 2, 0, 1, 2), (4, 1, 0, 64, 64)]
    assert Ops._chunk_parts([3, 2], 1 << 20) == [(0, 2, 0, 3, 5)]
