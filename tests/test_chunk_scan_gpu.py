"""Recurrences over a matrix state chunk by chunk, at the edges of chunks, heads and windows:
against float64 token by token, and no further from it than the token-by-token kernels."""

from types import SimpleNamespace

import pytest
import torch

from mini_llm_stack_b200.ops.kernels import Runtime

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    o = Runtime("cuda:0", torch.bfloat16).ops
    o.require_part("scan")
    o.require_part("mlstm")
    return o


def a_step(lens, chunked):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    slots = [(3 * r + 1) % len(lens) if len(lens) % 3 else r for r in range(len(lens))]
    i32 = dict(dtype=torch.int32, device="cuda")
    return SimpleNamespace(n_tokens=cu[-1], n_requests=len(lens), cu_q=torch.tensor(cu, **i32),
                           state_slot=torch.tensor(slots, **i32), q_lens=lens if chunked else []), cu, slots


def closer(got, other, want, chain, what):
    """``got`` lies no further from ``want`` than one and a half times ``other`` (both float32), or
    than a walk of ``chain`` roundings of 2^-24 takes a sum (one chunk's sums are one chain, the
    token-by-token kernels add eight shorter ones)."""
    scale = want.abs().max()
    mine, theirs = (got.double() - want).norm(), (other.double() - want).norm()
    assert torch.isfinite(got).all(), what
    assert mine <= max(1.5 * theirs, 2.0 ** -24 * chain ** 0.5 * want.norm()), (what, float(mine / want.norm()), float(theirs / want.norm()))
    assert (got.double() - want).abs().max() <= 2e-5 * scale, what


@pytest.fixture
def always(ops, monkeypatch):
    monkeypatch.setattr(ops, "CHUNKED_FROM", {"head": 1, "token": 1, "mlstm": 1}, raising=False)
    monkeypatch.setattr(ops, "CHUNK_TOKENS", 0, raising=False)
    return monkeypatch


LENS = [[1], [63, 64, 65], [130, 1, 7, 128], [300]]


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("e, f, heads", [(16, 16, 2), (64, 64, 3), (96, 200, 2), (128, 256, 2), (68, 132, 1), (256, 36, 1)])
@pytest.mark.parametrize("kind", ["head", "head_silu", "token", "token_plain"])
def test_linear_scan(ops, always, lens, e, f, heads, kind):
    if kind.startswith("token") and e > 128:
        pytest.skip("token by token")
    g = torch.Generator().manual_seed(e + f + sum(lens))
    t = sum(lens)
    q, k = (torch.randn(t, heads * e, generator=g) * e ** -0.5 for _ in range(2))
    v = torch.randn(t, heads * f, generator=g).bfloat16()
    if kind == "head_silu":
        q, k = q.bfloat16(), k.bfloat16()
    state0 = torch.randn(len(lens), heads * e * f, generator=g)
    # decays from nothing at all to everything, most of them close to one
    every = torch.cat([torch.tensor([0.0, 1.0, 1e-30, 0.5]), 1 - 2.0 ** -(1 + 7 * torch.rand(4096, generator=g))])
    head = kind.startswith("head")
    decay_head = every[torch.randint(0, 8 if heads > 1 else 4096, (heads,), generator=g)]
    decay_tok = every[torch.randint(0, 400, (t, heads * e), generator=g)].contiguous()
    bonus = torch.randn(heads, e, generator=g).bfloat16() if kind == "token" else None
    act = torch.nn.functional.silu if kind == "head_silu" else (lambda x: x)
    outs = {}
    for chunked in (True, False):
        step, cu, slots = a_step(lens, chunked)
        state = state0.cuda()
        out = torch.full((t, heads * f), float("nan"), device="cuda")
        before = ops.launches
        ops.linear_scan((q.cuda(), 0), (k.cuda(), 0), (v.cuda(), 0), state, step, heads, e, f, out,
                        decay_tok=None if head else decay_tok.cuda(),
                        decay_head=decay_head.cuda() if head else None,
                        bonus=None if bonus is None else bonus.cuda(), read_first=not head,
                        silu=kind == "head_silu")
        assert (ops.launches - before > 1) == chunked
        outs[chunked] = out.cpu(), state.cpu()
    want, last = torch.zeros(t, heads, f, dtype=torch.float64), torch.zeros(len(lens), heads, e, f, dtype=torch.float64)
    qd, kd, vd = (act(x.double()).view(t, heads, -1) for x in (q, k, v))
    for r, n in enumerate(lens):
        s = state0[slots[r]].double().view(heads, e, f)
        for i in range(cu[r], cu[r] + n):
            kv = kd[i][:, :, None] * vd[i][:, None, :]
            if head:
                s = decay_head.double()[:, None, None] * s + kv
                want[i] = torch.einsum("hef,he->hf", s, qd[i])
            else:
                u = bonus.double()[:, :, None] if bonus is not None else 0.0
                want[i] = torch.einsum("hef,he->hf", s + u * kv, qd[i])
                s = decay_tok[i].double().view(heads, e, 1) * s + kv
        last[slots[r]] = s
    closer(outs[True][0], outs[False][0], want.view(t, -1), e + 64, "outputs")
    closer(outs[True][1], outs[False][1], last.view(len(lens), -1), 64, "states")


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("e, f, heads", [(16, 64, 2), (64, 192, 2), (96, 192, 1), (256, 512, 1)])
@pytest.mark.parametrize("forget", [3.0, -4.0])
def test_mlstm(ops, always, lens, e, f, heads, forget):
    g = torch.Generator().manual_seed(e + f + sum(lens))
    t, width = sum(lens), ops.mlstm_state_width(e, f)
    qkv = torch.randn(t, heads * (2 * e + f), generator=g).bfloat16()
    gates = torch.randn(t, 2 * heads, generator=g) * 4.0
    bi, bf = torch.randn(heads, generator=g), torch.randn(heads, generator=g) + forget
    state0 = torch.randn(len(lens), heads, width, generator=g) * 0.3
    state0[:, :, e * f + e:] = state0[:, :, e * f + e:e * f + e + 1]
    outs = {}
    for chunked in (True, False):
        step, cu, slots = a_step(lens, chunked)
        state, num, den = state0.cuda(), torch.empty(t, heads * f, device="cuda"), torch.empty(t, heads, device="cuda")
        before = ops.launches
        ops.mlstm_scan(qkv.cuda(), (0, heads * e, 2 * heads * e), gates.cuda(), bi.cuda(), bf.cuda(), 15.0, step,
                       state, heads, e, f, num, den)
        assert (ops.launches - before > 1) == chunked
        outs[chunked] = num.cpu(), den.cpu(), state.cpu()
    q, k, v = (x.double().view(t, heads, -1) for x in qkv.split([heads * e, heads * e, heads * f], 1))
    q = q * e ** -0.5
    ig = 15 * torch.tanh((gates[:, :heads].double() + bi.double()) / 15)
    fg = torch.nn.functional.logsigmoid(15 * torch.tanh((gates[:, heads:].double() + bf.double()) / 15))
    want, last = torch.zeros(t, heads, f, dtype=torch.float64), state0.double().clone()
    want_den = torch.zeros(t, heads, dtype=torch.float64)
    for r, n in enumerate(lens):
        st = state0[slots[r]].double()
        c, norm, m = st[:, :e * f].reshape(heads, e, f).clone(), st[:, e * f:e * f + e].clone(), st[:, e * f + e].clone()
        for i in range(cu[r], cu[r] + n):
            new = torch.maximum(fg[i] + m, ig[i])
            keep, take = torch.exp(fg[i] + m - new), torch.exp(ig[i] - new)
            m = new
            c = keep[:, None, None] * c + (take[:, None] * k[i])[:, :, None] * v[i][:, None, :]
            norm = keep[:, None] * norm + take[:, None] * k[i]
            want_den[i] = torch.maximum((norm * q[i]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            want[i] = torch.einsum("hef,he->hf", c, q[i])
        last[slots[r], :, :e * f] = c.reshape(heads, -1)
        last[slots[r], :, e * f:e * f + e] = norm
        last[slots[r], :, e * f + e:] = m[:, None]
    # (a stabiliser of up to 16 is rounded to float32, which scales both by up to 16 * 2^-24)
    for got, other, exact in zip(outs[True], outs[False], (want.view(t, -1), want_den, last)):
        closer(got, other, exact, e + 64 + 16 ** 2, "numerators, denominators, states")


def test_windows_of_chunks_and_portions_go_on_from_the_slot(ops, always):
    """Scratch for one chunk a request at a time, and a prompt in two steps: the same states."""
    g = torch.Generator().manual_seed(5)
    lens, heads, e, f = [200, 70, 3], 2, 64, 64
    t = sum(lens)
    q, k, v = (torch.randn(t, heads * e, generator=g).bfloat16().cuda() for _ in range(3))
    decay = torch.tensor([0.97, 0.6]).cuda()

    def walk(lens, rows, state):
        step, _, _ = a_step(lens, True)
        step.state_slot = torch.arange(len(lens), dtype=torch.int32, device="cuda")
        out = torch.empty(sum(lens), heads * f, device="cuda")
        ops.linear_scan(*(((x[rows].contiguous(), 0)) for x in (q, k, v)), state, step, heads, e, f, out,
                        decay_head=decay)
        return out

    every = torch.arange(t, device="cuda")
    whole = torch.zeros(3, heads * e * f, device="cuda")
    out = walk(lens, every, whole)
    always.setattr(ops, "CHUNK_SCRATCH", 1, raising=False)
    cut = torch.zeros(3, heads * e * f, device="cuda")
    assert torch.equal(walk(lens, every, cut), out) and torch.equal(cut, whole)
    first, second = [100, 64, 1], [100, 6, 2]
    starts = [0, 200, 270]
    two = torch.zeros(3, heads * e * f, device="cuda")
    a = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, first)]).cuda()
    b = torch.cat([torch.arange(s + m, s + m + n) for s, m, n in zip(starts, first, second)]).cuda()
    got = torch.empty_like(out)
    got[a], got[b] = walk(first, a, two), walk(second, b, two)
    assert (got - out).abs().max() <= 1e-5 * out.abs().max() and (two - whole).abs().max() <= 1e-5 * whole.abs().max()


@pytest.mark.parametrize("kind", ["head", "token", "mlstm"])
def test_a_requests_bits_do_not_depend_on_its_neighbours(ops, kind):
    """Requests on both sides of the line between the kernels, more of them than a warp's lanes, beside
    each other and alone: a request's own length says which kernel takes it."""
    lens = [1] * 30 + [47, 48, 1, 200, 127, 128, 5, 65, 1, 191, 192]
    heads, e, f = 2, 64, 128
    t, r = sum(lens), len(lens)
    g = torch.Generator().manual_seed(7)
    rows = torch.randn(t, heads * (2 * e + f), generator=g).bfloat16().cuda()
    decay_head = torch.tensor([0.97, 0.8]).cuda()
    decay_tok = (1 - 0.2 * torch.rand(t, heads * e, generator=g)).cuda()
    gates = torch.randn(t, 2 * heads, generator=g).cuda()
    bias = torch.randn(2, heads, generator=g).cuda()
    width = ops.mlstm_state_width(e, f) if kind == "mlstm" else e * f
    state0 = torch.randn(r, heads * width, generator=g).cuda()
    if kind == "mlstm":
        state0.view(r, heads, width)[:, :, e * f + e:] = 0.5

    def walk(lens, at, slots):
        n = sum(lens)
        x, step = rows[at:at + n].contiguous(), a_step(lens, True)[0]
        step.state_slot = torch.arange(len(lens), dtype=torch.int32, device="cuda")
        state = state0[slots].clone()
        out = torch.full((n, heads * f), float("nan"), device="cuda")
        den = torch.zeros(n, heads, device="cuda")
        before = ops.launches
        if kind == "mlstm":
            ops.mlstm_scan(x, (0, heads * e, 2 * heads * e), gates[at:at + n].contiguous(), bias[0], bias[1], 15.0,
                           step, state.view(len(lens), heads, width), heads, e, f, out, den)
        else:
            ops.linear_scan((x, 0), (x, heads * e), (x, 2 * heads * e), state, step, heads, e, f, out,
                            decay_tok=decay_tok[at:at + n].contiguous() if kind == "token" else None,
                            decay_head=decay_head if kind == "head" else None, read_first=kind == "token")
        return out, den, state, ops.launches - before

    whole, at = walk(lens, 0, slice(0, r)), 0
    assert torch.isfinite(whole[0]).all()
    short = 1 if kind == "mlstm" else 0
    assert whole[3] == 5 + short                       # the chunks' kernels and one for the other requests
    least = ops.CHUNKED_FROM[kind]
    for i, n in enumerate(lens):
        alone = walk([n], at, slice(i, i + 1))
        assert alone[3] == (4 + short if n >= least else 1)
        for x, y in zip(whole[:2], alone[:2]):
            assert torch.equal(x[at:at + n], y), (i, n)
        assert torch.equal(whole[2][i], alone[2][0]), (i, n)
        at += n


@pytest.mark.parametrize("kind, heads, e, f", [("head", 16, 128, 256), ("token", 32, 64, 64), ("mlstm", 4, 256, 512)])
@pytest.mark.parametrize("more", [0, 17, 300])
def test_no_further_from_float64_than_token_by_token(ops, kind, heads, e, f, more):
    """From the shortest request that goes chunk by chunk on, at the sizes and decays of real layers.
    Norms of two sets of n independent errors of the same size differ by chance by 1 / sqrt(n) of
    themselves or so (each varies by 1 / sqrt(2n)): twice that is allowed, which counts for the
    denominators only (4 a token), and a hundredth for errors that are not independent."""
    t = ops.CHUNKED_FROM[kind] + more
    g = torch.Generator(device="cuda").manual_seed(t)
    q, k, v = (torch.randn(t, heads * w, device="cuda", generator=g).bfloat16() for w in (e, e, f))
    head = torch.tensor([1 - 2.0 ** (-5 - 3 * i / heads) for i in range(heads)], device="cuda")
    pace = torch.rand(heads * e, device="cuda", generator=g) * 5 - 6
    tok = torch.exp(-torch.exp(pace + 0.3 * torch.randn(t, heads * e, device="cuda", generator=g)))
    bonus = (torch.randn(heads, e, device="cuda", generator=g) * 0.5).bfloat16()
    gates = torch.randn(t, 2 * heads, device="cuda", generator=g)
    bi, bf = torch.randn(heads, device="cuda", generator=g), torch.randn(heads, device="cuda", generator=g) + 3
    got = {}
    for chunked in (True, False):
        step = a_step([t], chunked)[0]
        out, den = torch.empty(t, heads * f, device="cuda"), torch.empty(t, heads, device="cuda")
        if kind == "mlstm":
            state = torch.zeros(1, heads, ops.mlstm_state_width(e, f), device="cuda")
            ops.mlstm_scan(torch.cat([q, k, v], 1), (0, heads * e, 2 * heads * e), gates, bi, bf, 15.0, step, state,
                           heads, e, f, out, den)
            got[chunked] = out, state[0, :, :e * f + e], den
        else:
            state = torch.zeros(1, heads * e * f, device="cuda")
            ops.linear_scan((q, 0), (k, 0), (v, 0), state, step, heads, e, f, out,
                            decay_tok=tok if kind == "token" else None, decay_head=head if kind == "head" else None,
                            bonus=bonus if kind == "token" else None, read_first=kind == "token")
            got[chunked] = out, state.view(heads, -1)
    q, k, v = (x.double().view(t, heads, -1) for x in (q, k, v))
    s, n, m = (torch.zeros(*x, dtype=torch.float64, device="cuda") for x in ((heads, e, f), (heads, e), (heads,)))
    ig = 15 * torch.tanh((gates[:, :heads].double() + bi.double()) / 15)
    fg = torch.nn.functional.logsigmoid(15 * torch.tanh((gates[:, heads:].double() + bf.double()) / 15))
    outs, dens = [], []
    for i in range(t):
        kv = k[i][:, :, None] * v[i][:, None, :]
        if kind == "head":
            s = head.double()[:, None, None] * s + kv
            outs.append(torch.einsum("hef,he->hf", s, q[i]))
        elif kind == "token":
            outs.append(torch.einsum("hef,he->hf", s + bonus.double()[:, :, None] * kv, q[i]))
            s = tok[i].double().view(heads, e, 1) * s + kv
        else:
            new = torch.maximum(fg[i] + m, ig[i])
            keep, take = torch.exp(fg[i] + m - new), torch.exp(ig[i] - new)
            m, s, n = new, keep[:, None, None] * s + take[:, None, None] * kv, keep[:, None] * n + take[:, None] * k[i]
            outs.append(torch.einsum("hef,he->hf", s, q[i]) * e ** -0.5)
            dens.append(torch.maximum((n * q[i]).sum(-1).abs() * e ** -0.5, torch.exp(-m)) + 1e-6)
    last = torch.cat([s.reshape(heads, -1), n], 1) if kind == "mlstm" else s.reshape(heads, -1)
    for i, want in enumerate([torch.stack(outs).view(t, -1), last] + ([torch.stack(dens)] if dens else [])):
        mine, theirs = ((got[x][i].double() - want).norm() / want.norm() for x in (True, False))
        assert mine <= (1.01 + 2 * want.numel() ** -0.5) * theirs, (i, float(mine), float(theirs))


@pytest.mark.parametrize("kind", ["head", "token", "mlstm"])
def test_scratch_is_bounded(always, kind):
    """Three chunks of scratch for 34 requests, and memory that gives out: parts of the work, the same bits."""
    ops = Runtime("cuda:0", torch.bfloat16).ops        # its own scratch
    for part in ("scan", "mlstm"):
        ops.require_part(part)
    always.setattr(ops, "CHUNKED_FROM", {"head": 2, "token": 2, "mlstm": 2}, raising=False)
    lens = [200, 70, 1, 600] + [3] * 30
    heads, e, f, t, r = 2, 64, 64, sum(lens), len(lens)
    g = torch.Generator().manual_seed(3)
    rows = torch.randn(t, heads * (2 * e + f), generator=g).bfloat16().cuda()
    decay = (1 - 0.2 * torch.rand(t, heads * e, generator=g)).cuda()
    gates, bias = torch.randn(t, 2 * heads, generator=g).cuda(), torch.randn(2, heads, generator=g).cuda()
    width = ops.mlstm_state_width(e, f) if kind == "mlstm" else e * f

    def walk():
        step = a_step(lens, True)[0]
        state = torch.zeros(r, heads * width, device="cuda")
        out, den = torch.full((t, heads * f), float("nan"), device="cuda"), torch.zeros(t, heads, device="cuda")
        if kind == "mlstm":
            ops.mlstm_scan(rows, (0, heads * e, 2 * heads * e), gates, bias[0], bias[1], 15.0, step,
                           state.view(r, heads, width), heads, e, f, out, den)
        else:
            ops.linear_scan((rows, 0), (rows, heads * e), (rows, 2 * heads * e), state, step, heads, e, f, out,
                            decay_tok=decay if kind == "token" else None,
                            decay_head=torch.tensor([0.97, 0.8]).cuda() if kind == "head" else None,
                            read_first=kind == "token")
        return out, den, state

    part = ops._part_lib("mlstm" if kind == "mlstm" else "scan")
    chunk = part["scratch"](("head", "token", "mlstm").index(kind), heads, e, f, 1)
    always.setattr(ops, "CHUNK_SCRATCH", 3 * chunk, raising=False)
    bounded = walk()
    assert ops._scratch["chunk_scan"].numel() <= max(3 * chunk, 1 << 16)
    always.setattr(ops, "CHUNK_SCRATCH", 1 << 27, raising=False)
    real = ops.scratch

    def short(tag, n):
        if n > 5 * chunk:
            raise torch.cuda.OutOfMemoryError("no more")
        return real(tag, n)

    always.setattr(ops, "scratch", short)
    given_out = walk()
    assert chunk <= ops.CHUNK_SCRATCH <= 5 * chunk
    always.setattr(ops, "scratch", real)
    always.setattr(ops, "CHUNK_SCRATCH", 1 << 27, raising=False)
    whole = walk()
    for x, y, z in zip(bounded, given_out, whole):
        assert torch.equal(x, z) and torch.equal(y, z) and torch.isfinite(z).all()


@pytest.mark.parametrize("kind", ["head", "token", "mlstm"])
@pytest.mark.parametrize("what", ["v", "k", "q"])
@pytest.mark.parametrize("odd", [float("inf"), float("nan")])
@pytest.mark.parametrize("f", [64, 132])
def test_no_number_reaches_earlier_tokens_or_other_requests(ops, always, kind, what, odd, f):
    """One entry of one token that is infinite or not a number: earlier tokens of its chunk and other
    requests keep their bits, later ones are no numbers where the token-by-token kernel has none."""
    lens, bad, heads, e = [70, 200, 3], 70 + 100, 2, 64
    t = sum(lens)
    g = torch.Generator().manual_seed(5)
    clean = torch.randn(t, heads * (2 * e + f), generator=g).bfloat16().cuda()
    spoiled = clean.clone()
    spoiled[bad, {"q": 0, "k": heads * e, "v": 2 * heads * e}[what] + 5] = odd
    decay = (1 - 0.2 * torch.rand(t, heads * e, generator=g)).cuda()
    gates, bias = torch.randn(t, 2 * heads, generator=g).cuda(), torch.randn(2, heads, generator=g).cuda()
    got = {}
    for name, rows, chunked in (("clean", clean, True), ("odd", spoiled, True), ("tokens", spoiled, False)):
        step = a_step(lens, chunked)[0]
        out, den = torch.empty(t, heads * f, device="cuda"), torch.ones(t, heads, device="cuda")
        if kind == "mlstm":
            state = torch.zeros(3, heads, ops.mlstm_state_width(e, f), device="cuda")
            ops.mlstm_scan(rows, (0, heads * e, 2 * heads * e), gates, bias[0], bias[1], 15.0, step, state, heads,
                           e, f, out, den)
        else:
            state = torch.zeros(3, heads * e * f, device="cuda")
            ops.linear_scan((rows, 0), (rows, heads * e), (rows, 2 * heads * e), state, step, heads, e, f, out,
                            decay_tok=decay if kind == "token" else None,
                            decay_head=torch.tensor([0.97, 0.8]).cuda() if kind == "head" else None,
                            read_first=kind == "token")
        got[name] = torch.cat([out, den], 1)
    untouched = torch.ones(t, dtype=torch.bool, device="cuda")
    untouched[bad:270] = False
    assert torch.equal(got["odd"][untouched], got["clean"][untouched])
    # (a denominator that is no number falls to its floor, in either kernel: the numerators tell)
    odd, tokens = (got[x][:, :heads * f].isfinite() for x in ("odd", "tokens"))
    assert torch.equal(odd, tokens) and not odd[bad].all()


@pytest.mark.parametrize("kind", ["head", "head_silu"])
@pytest.mark.parametrize("e, f, heads", [(64, 128, 2), (160, 300, 1), (252, 516, 1)])
def test_wide_heads_on_tensor_cores(ops, always, e, f, heads, kind):
    """Heads of one, two and four groups of 128 columns a block, with remainders of 64 rows and of 128 columns."""
    test_linear_scan(ops, always, [130, 1, 7, 128], e, f, heads, kind)


def test_small_values_keep_their_bits(ops, always):
    """Values (and so the state) whose lower bfloat16 parts lie below bfloat16's smallest number: the outputs
    are those of ordinary values times a power of two."""
    heads, e, f, lens = 2, 128, 256, [130, 64]
    g = torch.Generator().manual_seed(11)
    t = sum(lens)
    q, k = (torch.randn(t, heads * e, generator=g).cuda() for _ in range(2))
    v = torch.randn(t, heads * f, generator=g).cuda()
    decay = torch.tensor([0.97, 0.6]).cuda()
    outs, states = [], []
    for power in (0, -116):
        step, _, _ = a_step(lens, True)
        state, out = torch.zeros(2, heads * e * f, device="cuda"), torch.empty(t, heads * f, device="cuda")
        ops.linear_scan((q, 0), (k, 0), (v * 2.0 ** power, 0), state, step, heads, e, f, out,
                        decay_head=decay)
        for to, x in ((outs, out), (states, state)):
            to.append(x.double() * 2.0 ** -power)
    # (float32's smallest, 2^-149, is 2^-33 of the values)
    assert (outs[1] - outs[0]).norm() <= 2.0 ** -23 * outs[0].norm()
    assert (states[1] - states[0]).norm() <= 2.0 ** -23 * states[0].norm()


@pytest.mark.parametrize("kind", ["head", "mlstm"])
def test_a_value_that_is_no_number_does_not_hold_a_prompt_up(ops, kind):
    """All tokens behind it are taken again: at most nine times the time (four; an output at a time
    took fourteen and seventeen)."""
    heads, e, f, t = 8, 128, 256, 2048
    rows = torch.randn(t, heads * (2 * e + f), device="cuda").bfloat16()
    odd = rows.clone()
    odd[10] = float("nan")
    gates, bias = torch.randn(t, 2 * heads, device="cuda"), torch.randn(2, heads, device="cuda")
    odd_gates = gates.clone()
    odd_gates[10] = float("nan")
    out, den, step = torch.empty(t, heads * f, device="cuda"), torch.empty(t, heads, device="cuda"), a_step([t], True)[0]

    def time(rows, gates):
        best = float("inf")
        for _ in range(4):
            state = torch.zeros(1, heads * (ops.mlstm_state_width(e, f) if kind == "mlstm" else e * f), device="cuda")
            begin, end = torch.cuda.Event(True), torch.cuda.Event(True)
            begin.record()
            if kind == "mlstm":
                ops.mlstm_scan(rows, (0, heads * e, 2 * heads * e), gates, bias[0], bias[1], 15.0, step,
                               state.view(1, heads, -1), heads, e, f, out, den)
            else:
                ops.linear_scan((rows, 0), (rows, heads * e), (rows, 2 * heads * e), state, step, heads, e, f, out,
                                decay_head=torch.full((heads,), 0.97, device="cuda"))
            end.record()
            torch.cuda.synchronize()
            best = min(best, begin.elapsed_time(end))
        return best
    plain = time(rows, gates)
    assert out.isfinite().all()
    assert time(odd, odd_gates) <= 9 * plain
    assert out[:10].isfinite().all() and out[10:].isnan().all()
