"""Attention without tensor cores: requests of several tokens go by tiles that share their keys, and
give the bits that a warp a row gives."""

from types import SimpleNamespace

import pytest
import torch

from mini_llm_stack_b200.ops.kernels import Runtime
from mini_llm_stack_b200.parts.base import GroupView

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd, heads, kv, block", [(16, 4, 2, 4), (64, 32, 8, 16), (20, 3, 1, 8), (80, 5, 5, 16),
                                                  (128, 72, 1, 32), (124, 4, 2, 16)])
@pytest.mark.parametrize("what", ["causal", "window", "keep", "chunk", "cap", "slopes"])
def test_tiles_give_the_bits_of_rows(act, hd, heads, kv, block, what):
    ops = Runtime("cuda:0", act).ops
    g = torch.Generator(device="cuda").manual_seed(hd + heads)
    lens, before = [1, 40, 7, 8, 70, 2, 33], [90, 0, 33, 25, 61, 0, 200]
    t, r = sum(lens), len(lens)
    most = max(b + n for b, n in zip(before, lens))
    width = -(-most // block)
    order = torch.randperm(r * width, generator=torch.Generator().manual_seed(1)).int()
    i32 = dict(dtype=torch.int32, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    pos = torch.cat([torch.arange(b, b + n) for b, n in zip(before, lens)])
    step = SimpleNamespace(n_tokens=t, n_requests=r, positions=pos.to(**i32), cu_q=torch.tensor(cu, **i32),
                           req_of_token=torch.repeat_interleave(torch.arange(r), torch.tensor(lens)).to(**i32),
                           groups={0: GroupView(order.view(r, width).to("cuda"), None, block, width)})
    pools = [torch.randn(kv, r * width, block, hd, device="cuda", generator=g).to(act) for _ in range(2)]
    cache = SimpleNamespace(group=0, k_pool=pools[0], v_pool=pools[1])
    # what no row may read: the places past every request's last token
    for i, (b, n) in enumerate(zip(before, lens)):
        for j in range(b + n, width * block):
            for p in pools:
                p[:, int(order[i * width + j // block]), j % block] = float("nan")
    qkv = torch.randn(t, (heads + 2 * kv) * hd, device="cuda", generator=g).to(act)
    args = dict(window=0)
    if what in ("window", "keep"):
        args = dict(window=37, keep_first=5 if what == "keep" else 0)
    if what == "chunk":
        args = dict(window=0, chunk=50)
    if what == "cap":
        args.update(softcap=2.0, sink=torch.randn(heads, device="cuda", generator=g))
    if what == "slopes":
        args.update(slopes=torch.rand(heads, device="cuda", generator=g))
    outs = []
    for q_lens in (lens, []):
        step.q_lens = q_lens
        out = torch.full((t, heads * hd), float("nan"), dtype=act, device="cuda")
        launches = ops.launches
        ops.paged_attention(qkv, out, cache, step, heads, kv, hd, hd ** -0.5, simt=True, **args)
        assert ops.launches - launches == (2 if q_lens else 1)
        outs.append(out)
    assert torch.isfinite(outs[1]).all() and torch.equal(outs[0], outs[1])
