"""Prompt attention where one cached row is key and value, on the tensor cores: against the kernel
of one warp a row, at the edges of key tiles (96), row tiles (128), pages, windows and chunks."""

from types import SimpleNamespace

import pytest
import torch

from mini_llm_stack_b200.ops.kernels import Runtime
from mini_llm_stack_b200.parts.attention import plan_paged_attention
from mini_llm_stack_b200.parts.base import GroupView

pytestmark = pytest.mark.gpu
HD = 256


@pytest.fixture(scope="module")
def ops():
    o = Runtime("cuda:0", torch.bfloat16).ops
    o.require_attention(HD)
    return o


@pytest.mark.parametrize("heads, block", [(16, 16), (32, 8), (3, 32), (5, 64)])
@pytest.mark.parametrize("lens, before, scattered", [
    ([1, 95, 2, 130], [95, 0, 300, 0], True), ([300], [0], False), ([33, 64], [700, 96], True),
    ([96, 97], [0, 95], False)])
@pytest.mark.parametrize("args", [dict(window=0), dict(window=100), dict(window=0, chunk=70), dict(window=33)])
@pytest.mark.parametrize("sinks", [False, True])
def test_against_a_warp_a_row(ops, monkeypatch, heads, block, lens, before, scattered, args, sinks):
    g = torch.Generator(device="cuda").manual_seed(heads + sum(lens))
    t, r = sum(lens), len(lens)
    ctx = [b + n for b, n in zip(before, lens)]
    width = -(-max(ctx) // block)
    order = (torch.randperm(r * width, generator=torch.Generator().manual_seed(1)) if scattered
             else torch.arange(r * width)).int()
    table = order.view(r, width).clone()
    for i, c in enumerate(ctx):
        table[i, -(-c // block):] = -1                   # pages that the request does not hold
        if args["window"]:                               # and those that a window has given back
            table[i, :max(0, before[i] - args["window"] + 1) // block] = -1
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device="cuda")
    step = SimpleNamespace(
        n_tokens=t, n_requests=r, q_lens=lens, ctx_lens=ctx, max_ctx_len=max(ctx), attn_tiles={},
        positions=torch.cat([torch.arange(b, c) for b, c in zip(before, ctx)]).to(**i32),
        cu_q=torch.tensor(cu, **i32), ctx_len=torch.tensor([*ctx, max(ctx)], **i32),
        req_of_token=torch.repeat_interleave(torch.arange(r), torch.tensor(lens)).to(**i32),
        groups={0: GroupView(table.cuda(), None, block, width)})
    pool = torch.randn(1, r * width, block, HD, device="cuda", generator=g).bfloat16()
    for i, c in enumerate(ctx):                          # the rest of a request's last page is cleared
        if c % block:
            pool[0, int(order[i * width + c // block]), c % block:] = 0.0
    cache = SimpleNamespace(group=0, k_pool=pool, v_pool=pool)
    qkv = torch.randn(t, (heads + 2) * HD, device="cuda", generator=g).bfloat16()
    qkv[:, :HD] *= 4.0                                   # a head whose softmax is nearly one key
    sink = torch.randn(heads, device="cuda", generator=g) * 2 if sinks else None
    facts = dict(ops.attention_facts(HD))
    plan = plan_paged_attention(step, facts, heads, 1, HD)
    got = {}
    for impl in ("auto", "simt"):
        monkeypatch.setattr(ops, "attention_impl", impl)
        out = torch.full((t, heads * HD), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(qkv, out, cache, step, heads, 1, HD, HD ** -0.5, plan=plan, sink=sink, **args)
        ops.check_status()
        got[impl] = out.float()
    assert torch.isfinite(got["auto"]).all()
    # outputs are averages of unit rows: P is rounded to 8 bits (2^-9 of a sum of weights at most 1,
    # times values of up to some 4), the result once more
    assert (got["auto"] - got["simt"]).abs().max() <= 2.0 ** -9 * 4 + 2.0 ** -8 * got["simt"].abs().max()


def test_every_tile_ends(ops):
    """Tiles of one to eight steps, many times over: the end of a tile is told by a barrier of its own,
    so that no wait looks for a phase that two later ones have passed.  The same bits every time."""
    lens, heads, block = [96 * n - 3 for n in range(1, 9)], 8, 16
    t, r = sum(lens), len(lens)
    width = -(-max(lens) // block)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device="cuda")
    step = SimpleNamespace(
        n_tokens=t, n_requests=r, q_lens=lens, ctx_lens=lens, max_ctx_len=max(lens), attn_tiles={},
        positions=torch.cat([torch.arange(n) for n in lens]).to(**i32),
        cu_q=torch.tensor(cu, **i32), ctx_len=torch.tensor([*lens, max(lens)], **i32),
        req_of_token=torch.repeat_interleave(torch.arange(r), torch.tensor(lens)).to(**i32),
        groups={0: GroupView(torch.arange(r * width, **i32).view(r, width), None, block, width)})
    g = torch.Generator(device="cuda").manual_seed(3)
    pool = torch.randn(1, r * width, block, HD, device="cuda", generator=g).bfloat16()
    cache = SimpleNamespace(group=0, k_pool=pool, v_pool=pool)
    qkv = torch.randn(t, (heads + 2) * HD, device="cuda", generator=g).bfloat16()
    plan = plan_paged_attention(step, dict(ops.attention_facts(HD)), heads, 1, HD)
    first = None
    for _ in range(200):
        out = torch.full((t, heads * HD), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(qkv, out, cache, step, heads, 1, HD, HD ** -0.5, 0, plan=plan)
        first = out if first is None else first
        assert torch.equal(out, first)
    ops.check_status()


@pytest.mark.parametrize("peak", [1.0, 2.0, 5.0])
@pytest.mark.parametrize("heads, kv", [(8, 1), (6, 2)])
def test_no_further_from_float64_than_the_tiles_it_replaces(ops, monkeypatch, peak, heads, kv):
    """Flat and peaked weights (scores of deviation ``peak``), beside the mma.sync tiles."""
    lens, block = [700, 45], 16
    t, r = sum(lens), len(lens)
    width = -(-max(lens) // block)
    i32 = dict(dtype=torch.int32, device="cuda")
    order = torch.randperm(r * width, generator=torch.Generator().manual_seed(2)).view(r, width)
    step = SimpleNamespace(
        n_tokens=t, n_requests=r, q_lens=lens, ctx_lens=lens, max_ctx_len=max(lens), attn_tiles={},
        positions=torch.cat([torch.arange(n) for n in lens]).to(**i32),
        cu_q=torch.tensor([0, lens[0], t], **i32), ctx_len=torch.tensor([*lens, max(lens)], **i32),
        req_of_token=torch.repeat_interleave(torch.arange(r), torch.tensor(lens)).to(**i32),
        groups={0: GroupView(order.to(**i32), None, block, width)})
    g = torch.Generator(device="cuda").manual_seed(heads)
    rows = torch.randn(kv, t, HD, device="cuda", generator=g).bfloat16()
    pool = torch.zeros(kv, r * width, block, HD, dtype=torch.bfloat16, device="cuda")
    at = 0
    for i, n in enumerate(lens):
        for j in range(n):
            pool[:, int(order[i, j // block]), j % block] = rows[:, at + j]
        at += n
    cache = SimpleNamespace(group=0, k_pool=pool, v_pool=pool)
    qkv = torch.randn(t, (heads + 2 * kv) * HD, device="cuda", generator=g).mul_(peak).bfloat16()
    plan = plan_paged_attention(step, dict(ops.attention_facts(HD)), heads, kv, HD)
    want, at = torch.empty(t, heads, HD, dtype=torch.float64, device="cuda"), 0
    for n in lens:
        hidden = torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1)
        for h in range(heads):
            k = rows[h // (heads // kv), at:at + n].double()
            s = qkv[at:at + n, h * HD:(h + 1) * HD].double() @ k.T * HD ** -0.5
            want[at:at + n, h] = torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ k
        at += n
    far = {}
    for impl in ("auto", "mma"):
        monkeypatch.setattr(ops, "attention_impl", impl)
        out = torch.full((t, heads * HD), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(qkv, out, cache, step, heads, kv, HD, HD ** -0.5, 0, plan=plan)
        far[impl] = float((out.double().view_as(want) - want).norm() / want.norm())
    ops.check_status()
    print(heads, kv, peak, far)
    assert far["auto"] <= 1.01 * far["mma"], far          # both are rounded to 8 bits once, which is most of it


def prompts(ops, heads=4, kv=1, lens=(130, 40), block=16):
    """A step of whole prompts over pages in order: (step, cache, qkv, plan)."""
    t, r = sum(lens), len(lens)
    width = -(-max(lens) // block)
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    step = SimpleNamespace(
        n_tokens=t, n_requests=r, q_lens=list(lens), ctx_lens=list(lens), max_ctx_len=max(lens), attn_tiles={},
        positions=torch.cat([torch.arange(n) for n in lens]).to(**i32),
        cu_q=torch.tensor(cu, **i32), ctx_len=torch.tensor([*lens, max(lens)], **i32),
        req_of_token=torch.repeat_interleave(torch.arange(r), torch.tensor(lens)).to(**i32),
        groups={0: GroupView(torch.arange(r * width, **i32).view(r, width), None, block, width)})
    g = torch.Generator(device="cuda").manual_seed(11)
    pool = torch.randn(kv, r * width, block, HD, device="cuda", generator=g).bfloat16()
    qkv = torch.randn(t, (heads + 2 * kv) * HD, device="cuda", generator=g).bfloat16()
    plan = plan_paged_attention(step, dict(ops.attention_facts(HD)), heads, kv, HD)
    return step, SimpleNamespace(group=0, k_pool=pool, v_pool=pool), qkv, plan


@pytest.fixture
def taken(ops, monkeypatch):
    """Calls that the kernel for shared rows took."""
    takes, fn = ops._attention_shared[HD]
    calls = []

    def counted(*args):
        calls.append(args)
        return fn(*args)

    monkeypatch.setitem(ops._attention_shared, HD, (takes, counted))
    return calls


def by_warps(ops, monkeypatch, step, cache, qkv, heads, kv, scale):
    with monkeypatch.context() as m:
        m.setattr(ops, "attention_impl", "simt")
        out = torch.empty(step.n_tokens, heads * HD, dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(qkv, out, cache, step, heads, kv, HD, scale, 0)
    return out.float()


@pytest.mark.parametrize("first", [0, 4, 8, 12])
def test_columns_of_a_wider_buffer(ops, monkeypatch, taken, first):
    """Output rows that start between 16-byte addresses are the mma.sync tiles'."""
    heads, scale = 4, HD ** -0.5
    step, cache, qkv, plan = prompts(ops, heads)
    wide = torch.full((step.n_tokens, heads * HD + 16), 7.0, dtype=torch.bfloat16, device="cuda")
    out = wide[:, first:first + heads * HD]
    ops.paged_attention(qkv, out, cache, step, heads, 1, HD, scale, 0, plan=plan)
    ops.check_status()
    assert len(taken) == (1 if first % 8 == 0 else 0)
    want = by_warps(ops, monkeypatch, step, cache, qkv, heads, 1, scale)
    assert (out.float() - want).abs().max() <= 2.0 ** -9 * 4 + 2.0 ** -8 * want.abs().max()
    assert (wide[:, :first] == 7.0).all() and (wide[:, first + heads * HD:] == 7.0).all()


@pytest.mark.parametrize("scale", [0.0, -0.0625])
def test_scales_that_are_not_positive(ops, monkeypatch, taken, scale):
    """The kernel takes the maximum of scores before they are scaled: such calls are the tiles'."""
    step, cache, qkv, plan = prompts(ops)
    out = torch.full((step.n_tokens, 4 * HD), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(qkv, out, cache, step, 4, 1, HD, scale, 0, plan=plan)
    ops.check_status()
    want = by_warps(ops, monkeypatch, step, cache, qkv, 4, 1, scale)
    assert (out.float() - want).abs().max() <= 2.0 ** -9 * 4 + 2.0 ** -8 * want.abs().max()
    assert not taken


@pytest.mark.parametrize("block, calls", [(8, 1), (16, 1), (32, 1), (64, 0)])
@pytest.mark.parametrize("heads, kv", [(4, 1), (6, 2)])
def test_which_pages_the_kernel_takes(ops, monkeypatch, taken, block, calls, heads, kv):
    step, cache, qkv, plan = prompts(ops, heads, kv, block=block)
    out = torch.full((step.n_tokens, heads * HD), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(qkv, out, cache, step, heads, kv, HD, HD ** -0.5, 0, plan=plan)
    ops.check_status()
    assert len(taken) == calls
    want = by_warps(ops, monkeypatch, step, cache, qkv, heads, kv, HD ** -0.5)
    assert (out.float() - want).abs().max() <= 2.0 ** -9 * 4 + 2.0 ** -8 * want.abs().max()


def test_rows_of_keys_and_values_apart_are_not_taken(ops, taken):
    step, cache, qkv, plan = prompts(ops)
    cache.v_pool = cache.k_pool.clone()
    out = torch.empty(step.n_tokens, 4 * HD, dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(qkv, out, cache, step, 4, 1, HD, HD ** -0.5, 0, plan=plan)
    ops.check_status()
    assert not taken
