"""The row kernels around the scans where rows are read four entries at a time and where they are
not: against float64."""

from types import SimpleNamespace

import pytest
import torch

from mini_llm_stack_b200.ops.kernels import Runtime

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    o = Runtime("cuda:0", torch.bfloat16).ops
    for part in ("scan", "mlstm", "shortconv"):
        o.require_part(part)
    return o


def near(got, want, act, terms=64):
    """One rounding to the type, behind float32 sums and functions of a few units of 2^-24."""
    unit = 2.0 ** -8 if act == torch.bfloat16 else 2.0 ** -22 * terms ** 0.5
    assert ((got.double() - want).abs() <= unit * want.abs() + 1e-6 * want.abs().max()).all()


@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("t, heads, f", [(1, 1, 4), (3, 5, 36), (9, 3, 128), (2, 3, 132), (7, 2, 256), (3, 3, 300),
                                         (1, 2, 512), (2, 2, 516), (5, 3, 30)])
@pytest.mark.parametrize("weighted", [False, True])
def test_finish(ops, act, t, heads, f, weighted):
    g = torch.Generator(device="cuda").manual_seed(t + f)
    o = torch.randn(t, heads * f, device="cuda", generator=g)
    gate = torch.randn(t, heads * f + 8, device="cuda", generator=g).to(act)
    w = (torch.rand(heads * f, device="cuda", generator=g) + 0.5).to(act)
    out = torch.full((t, heads * f), float("nan"), dtype=act, device="cuda")
    ops.scan_finish(o, gate, 8, w if weighted else None, 1e-5, out, heads, f)
    z, x = gate[:, 8:].double(), o.double().view(t, heads, f)
    n = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)).view(t, -1)
    near(out, n * (w.double() if weighted else 1.0) * z * torch.sigmoid(z), act, f)
    den = torch.rand(t, heads, device="cuda", generator=g) + 0.5
    ops.mlstm_finish(o, den, gate, 8, w, 1e-5, out, heads, f)
    x = x / den.double()[:, :, None]
    n = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)).view(t, -1)
    near(out, n * w.double() * torch.sigmoid(z), act, f)


@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("t, heads, e, dims", [(1, 1, 8, 8), (5, 3, 64, 32), (4, 2, 64, 60), (3, 32, 128, 128),
                                               (2, 3, 72, 8), (2, 5, 128, 0), (3, 2, 20, 8)])
def test_rotation(ops, act, t, heads, e, dims):
    rotation(ops, act, t, heads, e, dims)


@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("t, heads, e, dims", [(1, 64, 8, 8), (5, 8, 64, 32), (4, 9, 64, 56), (2, 8, 72, 8), (3, 7, 72, 72),
                                               (2, 4, 128, 0), (2, 26, 20, 8), (1, 1, 512, 256)])
def test_rotation_of_wide_rows(ops, act, t, heads, e, dims):
    """Rows on both sides of 512 entries, from which on they go four entries at a time."""
    rotation(ops, act, t, heads, e, dims)


def rotation(ops, act, t, heads, e, dims):
    g = torch.Generator(device="cuda").manual_seed(t + e)
    width = heads * e
    src = torch.randn(t, 3 * width, device="cuda", generator=g).to(act)
    pos = torch.randint(0, 5000, (t,), dtype=torch.int32, device="cuda", generator=g)
    freq = torch.pow(torch.tensor(1e4, dtype=torch.float64), -2.0 * torch.arange(dims // 2, dtype=torch.float64) / max(dims, 1)).cuda()
    out = torch.full((t, 2 * width), float("nan"), device="cuda")
    ops.rotate_rows(src, 0, 2 * width, pos, freq if dims else None, dims, 0.25, out, heads, e)
    a = pos.double()[:, None] * freq
    c, s = a.cos()[:, None], a.sin()[:, None]
    for got, x, scale in ((out[:, :width], src[:, :width], 1.0), (out[:, width:], src[:, 2 * width:], 0.25)):
        x = x.double().reshape(t, heads, e).clone()
        lo, hi = x[..., :dims // 2].clone(), x[..., dims // 2:dims].clone()
        x[..., :dims // 2], x[..., dims // 2:dims] = lo * c - hi * s, hi * c + lo * s
        assert (got.double() - scale * x.view(t, -1)).abs().max() <= 4e-6


@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d, rank", [(64, 4), (66, 6), (1028, 64), (300, 33)])
def test_shift_and_decay(ops, act, d, rank):
    g = torch.Generator(device="cuda").manual_seed(d)
    lens, t = [17, 1, 3], 21
    i32 = dict(dtype=torch.int32, device="cuda")
    step = SimpleNamespace(n_tokens=t, n_requests=3, cu_q=torch.tensor([0, 17, 18, 21], **i32),
                           req_of_token=torch.tensor([0] * 17 + [1] + [2] * 3, **i32),
                           state_slot=torch.tensor([2, 0, 1], **i32), q_lens=lens)
    h = torch.randn(t, d, device="cuda", generator=g).to(act)
    mu = torch.rand(3, d, device="cuda", generator=g).to(act)
    tail = torch.randn(3, d, device="cuda", generator=g)
    out = torch.full((2, t, d), float("nan"), dtype=act, device="cuda")
    last = torch.full((t, d), float("nan"), device="cuda")
    ops.token_shift_mix(h, mu, tail, out, last, step)
    prev = torch.cat([tail[2:3], h[:16].float(), tail[:1], tail[1:2], h[18:20].float()]).double()
    for s, got in enumerate((out[0], out[1], last)):
        want = h.double() + (prev - h.double()) * mu[s].double()
        near(got, want, act if s < 2 else torch.float32)
    lo = torch.randn(t, rank, device="cuda", generator=g)
    w2 = torch.randn(rank, d, device="cuda", generator=g) * 0.1
    w0 = torch.randn(d, device="cuda", generator=g).to(act)
    decay = torch.full((t, d), float("nan"), device="cuda")
    ops.decay_lowrank(lo, w2, w0, decay)
    want = torch.exp(-torch.exp(torch.tanh(lo.double()) @ w2.double() + w0.double()))
    assert (decay.double() - want).abs().max() <= 2e-6
