"""The experts' products on the tensor cores against float64, at the edges of their tiles: rows of
an expert around 16, 32, 128 and 256, outputs and inputs that fill no tile, experts without rows,
all rows at one expert, outputs that stand for no expert."""

import pytest
import torch

from mini_llm_stack_b200.ops.kernels import Runtime

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    o = Runtime("cuda:0", torch.bfloat16).ops
    o.require_part("experts")
    return o


def routed(ops, idx, weight, experts, n_real):
    """The arrays of a step in which token t takes the outputs idx[t] (weights for combining)."""
    t, top = idx.shape
    n, i32 = t * top, dict(dtype=torch.int32, device="cuda")
    tiles = ops.expert_max_tiles(n, experts)
    work = {"idx": torch.empty(n, **i32), "weight": torch.empty(n, device="cuda"),
            "order": torch.empty(n, **i32), "offsets": torch.empty(experts + 1, **i32),
            "cursor": torch.empty(experts, **i32), "tile_expert": torch.empty(tiles, **i32),
            "tile_row0": torch.empty(tiles, **i32), "max_tiles": tiles}
    logits = torch.full((t, experts), -50.0)
    logits.scatter_(1, idx, (torch.arange(top, 0, -1).float() + 3.0).expand(t, top))
    ops.route(logits.cuda(), top, False, work, n_real=n_real)
    assert torch.equal(work["idx"].cpu().view(t, top).long(), idx)
    work["weight"].copy_(weight.reshape(-1))
    return work


def choices(t, experts, top, spread, g):
    if spread == "one":                      # every token's first choice is the same expert
        idx = torch.stack([torch.randperm(experts - 1, generator=g)[:top] + 1 for _ in range(t)])
        idx[:, 0] = 0
        return idx
    return torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(t)])


CASES = [  # tokens, experts, identity outputs, top, d, f, spread
    (1, 3, 0, 1, 64, 16, "even"), (16, 4, 0, 1, 72, 40, "one"), (17, 4, 1, 2, 136, 128, "one"),
    (33, 5, 0, 2, 64, 136, "one"), (40, 2, 0, 1, 200, 129, "even"), (129, 3, 0, 2, 64, 96, "one"),
    (127, 2, 0, 2, 320, 264, "even"), (257, 3, 1, 2, 128, 72, "one"), (600, 4, 0, 1, 64, 130, "even"),
    (515, 2, 0, 1, 256, 384, "one"), (70, 300, 0, 3, 64, 32, "even")]


@pytest.mark.parametrize("t, experts, identity, top, d, f, spread", CASES)
@pytest.mark.parametrize("unit", ["silu", "clamped", "relu2"])
def test_products_of_sorted_rows(ops, t, experts, identity, top, d, f, spread, unit):
    g = torch.Generator().manual_seed(t + experts)
    outputs = experts + identity
    idx = choices(t, outputs, top, spread, g)
    weight = torch.rand(t, top, generator=g) + 0.1
    work = routed(ops, idx, weight, outputs, experts)
    h = torch.randn(t, d, generator=g).bfloat16()
    mats = 1 if unit == "relu2" else 2
    w1 = (torch.randn(experts, mats * f, d, generator=g) * d ** -0.5).bfloat16()
    w2 = (torch.randn(experts, d, f, generator=g) * f ** -0.5).bfloat16()
    n = t * top
    y = torch.full((n, f), float("nan"), dtype=torch.bfloat16, device="cuda")
    out = torch.full((n, d), float("nan"), device="cuda")
    scale_in = unit == "silu"
    if unit == "relu2":
        ops.expert_relu_squared(h.cuda(), w1.cuda(), y, work, top, scale_in)
    else:
        ops.expert_glu(h.cuda(), w1.cuda(), y, work, top, scale_in, alpha=1.702,
                       limit=0.5 if unit == "clamped" else 0.0)
    ops.expert_down(y, w2.cuda(), out, work, top, not scale_in)
    ops.check_status()
    order = work["order"].cpu().long()
    place = torch.empty(n, dtype=torch.long)
    place[order] = torch.arange(n)
    y, out = y.cpu(), out.cpu()
    for tok in range(t):
        for j in range(top):
            slot, e = tok * top + j, int(idx[tok, j])
            if e >= experts:
                continue
            a = h[tok].float() * weight[tok, j] if scale_in else h[tok].float()
            z = w1[e].double() @ a.bfloat16().double()
            if unit == "relu2":
                want = z.clamp(min=0) ** 2
            else:
                gate, up = z[:f], z[f:]
                if unit == "clamped":
                    gate, up = gate.clamp(max=0.5), up.clamp(-0.5, 0.5)
                    want = gate * torch.sigmoid(1.702 * gate) * (up + 1)
                else:
                    want = gate * torch.sigmoid(gate) * up
            row = y[place[slot]].double()
            # one rounding to 8 bits behind float32 sums of d products
            assert (row - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 1e-5, (tok, j)
            down = w2[e].double() @ row * (1.0 if scale_in else float(weight[tok, j]))
            # float32 sums of f products of unit size
            assert (out[slot].double() - down).abs().max() <= 1e-5 * max(1.0, float(row.norm())), (tok, j)


@pytest.mark.parametrize("experts, groups", [(5, None), (64, (8, 3)), (65, None), (256, (4, 1)), (257, None), (9000, None)])
def test_choice_and_order(ops, experts, groups):
    """Choices against a stable sort (scores of few distinct values, numbers that are none), and the
    slots in the order of their experts."""
    g = torch.Generator().manual_seed(experts)
    t, top = 37, min(5, experts)
    logits = torch.randint(-6, 7, (t, experts), generator=g).float()
    logits[3, 1] = float("nan")
    i32 = dict(dtype=torch.int32, device="cuda")
    n, tiles = t * top, ops.expert_max_tiles(t * top, experts)
    work = {"idx": torch.empty(n, **i32), "weight": torch.empty(n, device="cuda"), "order": torch.empty(n, **i32),
            "offsets": torch.empty(experts + 1, **i32), "cursor": torch.empty(experts, **i32),
            "tile_expert": torch.empty(tiles, **i32), "tile_row0": torch.empty(tiles, **i32), "max_tiles": tiles}
    ops.route(logits.cuda(), top, False, work, n_real=experts - 1, groups=groups)
    idx = work["idx"].cpu().view(t, top).long()
    for i in range(t):
        allowed = set(range(experts))
        if i == 3:
            allowed.discard(1)
        elif groups:
            size = experts // groups[0]
            best = logits[i].view(groups[0], size).sigmoid().topk(2, -1).values.sum(-1)
            keep = sorted(range(groups[0]), key=lambda k: (-float(best[k]), k))[:groups[1]]
            allowed = {e for e in allowed if e // size in keep}
        if i == 3 and groups:
            continue
        want = sorted(allowed, key=lambda e: (-float(logits[i, e]), e))[:top]
        assert idx[i].tolist() == want + [0] * (top - len(want)), i      # (no number left: output 0)
    offsets, order = work["offsets"].cpu(), work["order"].cpu().long()
    counts = torch.bincount(idx.reshape(-1), minlength=experts)
    assert torch.equal(offsets[1:] - offsets[:-1], counts.int()) and offsets[0] == 0
    assert torch.equal(order.sort().values, torch.arange(n))
    assert torch.equal(idx.reshape(-1)[order], torch.repeat_interleave(torch.arange(experts), counts))
    want = [(e, int(offsets[e]) + r) for e in range(experts - 1) for r in range(0, int(counts[e]), 32)]
    got = list(zip(work["tile_expert"].tolist(), work["tile_row0"].tolist()))
    assert got[:len(want)] == want and all(e == -1 for e, _ in got[len(want):])


@pytest.mark.parametrize("d", [4, 30, 64, 1028])
@pytest.mark.parametrize("top", [1, 6, 9])
@pytest.mark.parametrize("shared", [None, "rows", "gated"])
def test_combination(ops, d, top, shared):
    combination(ops, 11, d, top, shared)


@pytest.mark.parametrize("t, d", [(255, 256), (256, 256), (280, 252), (64, 1024), (63, 1024), (130, 516), (130, 514)])
@pytest.mark.parametrize("top", [1, 9])
@pytest.mark.parametrize("shared", [None, "rows", "gated"])
def test_combination_of_more_rows(ops, t, d, top, shared):
    """Both sides of the line from which on rows are added up four entries at a time."""
    combination(ops, t, d, top, shared)


def combination(ops, t, d, top, shared):
    g = torch.Generator().manual_seed(d + top)
    n_real = 7
    per_slot = torch.randn(t * top, d, generator=g)
    h = torch.randn(t, d, generator=g).bfloat16()
    idx = torch.randint(0, n_real + 2, (t, top), generator=g)
    weight = torch.rand(t, top, generator=g)
    rows = torch.randn(t, d, generator=g).bfloat16()
    gate = torch.randn(t, 3, generator=g)
    delta = torch.full((t, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    work = {"idx": idx.int().reshape(-1).cuda(), "weight": weight.reshape(-1).cuda()}
    ops.expert_combine(per_slot.cuda(), top, rows.cuda() if shared else None, delta, work=work, n_real=n_real,
                       h=h.cuda(), shared_gate=gate.cuda()[:, 2] if shared == "gated" else None)
    own = (idx >= n_real)[..., None]
    want = torch.where(own, weight.double()[..., None] * h.double()[:, None], per_slot.double().view(t, top, d)).sum(1)
    if shared:
        want = want + rows.double() * (torch.sigmoid(gate[:, 2:].double()) if shared == "gated" else 1.0)
    # float32 sums of `top` values, one rounding to 8 bits
    assert ((delta.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()


@pytest.mark.parametrize("unit", ["silu", "relu2"])
def test_more_experts_than_a_launch_takes(ops, unit):
    """5,000 experts, rows at both ends and on both sides of 4,096, on the tensor cores; a few rows of
    each against float64."""
    g = torch.Generator(device="cuda").manual_seed(1)
    experts, t, top, d, f = 5000, 40, 3, 64, 16
    idx = torch.randint(0, experts, (t, top), generator=torch.Generator().manual_seed(2))
    idx[:, 1] = (idx[:, 0] + 1) % experts
    idx[:, 2] = (idx[:, 0] + 2) % experts
    idx[:8] = torch.tensor([[0, 4095, 4096]] * 4 + [[4999, 4096, 1]] * 4)
    work = routed(ops, idx, torch.ones(t, top), experts, experts)
    h = torch.randn(t, d, device="cuda", generator=g).bfloat16()
    mats = 1 if unit == "relu2" else 2
    w1 = (torch.randn(experts, mats * f, d, device="cuda", generator=g) * d ** -0.5).bfloat16()
    w2 = (torch.randn(experts, d, f, device="cuda", generator=g) * f ** -0.5).bfloat16()
    assert ops._part_lib("experts")["takes_tc"](1, h.data_ptr(), w1.data_ptr(), d)
    n = t * top
    y = torch.full((n, f), float("nan"), dtype=torch.bfloat16, device="cuda")
    out = torch.full((n, d), float("nan"), device="cuda")
    (ops.expert_relu_squared if unit == "relu2" else ops.expert_glu)(h, w1, y, work, top, False)
    ops.expert_down(y, w2, out, work, top, False)
    ops.check_status()
    rows, e = torch.arange(n, device="cuda") // top, idx.reshape(-1).cuda()
    z = torch.einsum("nfd,nd->nf", w1[e].double(), h[rows].double())
    want = z.clamp(min=0) ** 2 if unit == "relu2" else z[:, :f] * torch.sigmoid(z[:, :f]) * z[:, f:]
    place = torch.empty(n, dtype=torch.long, device="cuda")
    place[work["order"].long()] = torch.arange(n, device="cuda")
    got = y[place].double()
    # one rounding to 8 bits behind float32 sums of d products; float32 sums of f products
    assert (got - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 1e-5
    down = torch.einsum("ndf,nf->nd", w2[e].double(), got)
    assert (out.double() - down).abs().max() <= 1e-5 * max(1.0, float(got.norm(dim=1).max()))


@pytest.mark.parametrize("t, experts, identity, top, d, f, spread", CASES)
def test_which_products_run_on_the_tensor_cores(ops, t, experts, identity, top, d, f, spread):
    """The cases above: rows of whole 16-byte pieces do (the gather of the first product is a launch more),
    the down products of 129 and 130 inputs do not."""
    idx = choices(t, experts + identity, top, spread, torch.Generator().manual_seed(0))
    work = routed(ops, idx, torch.ones(t, top), experts + identity, experts)
    b16 = dict(dtype=torch.bfloat16, device="cuda")
    h, y, out = torch.zeros(t, d, **b16), torch.zeros(t * top, f, **b16), torch.zeros(t * top, d, device="cuda")
    w1, w2 = torch.zeros(experts, 2 * f, d, **b16), torch.zeros(experts, d, f, **b16)
    takes = ops._part_lib("experts")["takes_tc"]
    assert d % 8 == 0 and takes(1, h.data_ptr(), w1.data_ptr(), d)
    assert bool(takes(1, y.data_ptr(), w2.data_ptr(), f)) == (f % 8 == 0)
    before = ops.launches
    ops.expert_glu(h, w1, y, work, top, True)
    assert ops.launches - before == 2
    ops.expert_down(y, w2, out, work, top, False)
    ops.check_status()
