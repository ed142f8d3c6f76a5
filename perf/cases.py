"""Measured cases: what programs built on this package run on the GPU, from one decoded token of a
small model to prompts of 2,048 tokens at the 8B sizes.

Whole calls go through ``ModelRunner.step`` (decoding) and ``ComposedModel.forward`` (prompts);
the other cases are single layers, a mixer or a feed-forward called as a block calls it, on rows
that a norm would have left (unit variance, bfloat16).  Weights are N(0, 0.02^2), the layer sizes
those of ``bench.py`` (``--shape``, ``--design``).  ``exact`` restates every case in float64.
"""

from __future__ import annotations

import math

import torch

from mini_llm_stack_b200.cache.manager import CacheManager
from mini_llm_stack_b200.config import config_from_dict
from mini_llm_stack_b200.config.registry import build_model
from mini_llm_stack_b200.engine.batch import BatchBuilder, Entry
from mini_llm_stack_b200.engine.runner import ModelRunner
from mini_llm_stack_b200.ops.kernels import Runtime
from mini_llm_stack_b200.parts.feedforward import RoutedExperts, SwiGLUFeedForward
from mini_llm_stack_b200.parts.latent_attention import LatentAttention
from mini_llm_stack_b200.parts.linear_recurrence import GatedDeltaMixer, RetentionMixer, WkvMixer
from mini_llm_stack_b200.parts.mlstm import MLstmMixer
from mini_llm_stack_b200.parts.position import PartialRotary

DEV = "cuda:0"
PAGE = 16
STD = 0.02
CONTEXT = 8192
EPS = 1e-5
GATE_CAP = 15.0

# Llama-3-8B and Llama-3.2-1B (bench.py --shape)
LLAMA = {
    "8b": dict(vocab_size=128256, d_model=4096, n_heads=32, n_kv_heads=8, head_dim=128,
               intermediate_size=14336, tie_embeddings=False),
    "1b": dict(vocab_size=128256, d_model=2048, n_heads=32, n_kv_heads=8, head_dim=64,
               intermediate_size=8192, tie_embeddings=True),
}
# the other architectures' layers (bench.py --design)
SIZES = {
    "1b": dict(width=2048, heads=16, dim=128, kv_rank=256, q_rank=768, experts=32, top=4,
               eff=1024, shared=1024, mheads=4, mdim=256, mvdim=512),
    "8b": dict(width=4096, heads=32, dim=128, kv_rank=256, q_rank=1536, experts=64, top=6,
               eff=1408, shared=2816, mheads=8, mdim=256, mvdim=512),
}
ROT_BASE = 1e6


# ------------------------------------------------------------------------------------- cases
def listed() -> list:
    return [
        # interactive serving of a few users with long contexts, one token each
        dict(name="llama_decode_8b_b8", kind="llama_decode", size="8b", layers=4, batch=8,
             context=8191),
        # one user of a small model: the latency of a token, all sixteen layers
        dict(name="llama_decode_1b_b1", kind="llama_decode", size="1b", layers=16, batch=1,
             context=1000),
        # a prompt comes in
        dict(name="llama_prompt_8b_2048", kind="llama_prompt", size="8b", layers=4, tokens=2048,
             requests=1, dtype="bfloat16"),
        # three prompts in the true float32 run that checks are made against
        dict(name="llama_prompt_1b_f32", kind="llama_prompt", size="1b", layers=2, tokens=515,
             requests=3, dtype="float32"),
        # a prompt through routed gated experts (weights on their inputs, a shared expert)
        dict(name="experts_8b_2048", kind="experts", size="8b", unit="gated", tokens=2048),
        # a short prompt through routed ungated experts (softmax over the chosen logits)
        dict(name="experts_1b_707", kind="experts", size="1b", unit="relu_squared", tokens=707),
        # decoded tokens of sixteen requests through the experts
        dict(name="experts_8b_16", kind="experts", size="8b", unit="gated", tokens=16),
        # prompts through attention over a cached latent
        dict(name="latent_8b_2048", kind="latent", size="8b", tokens=2048, requests=2),
        # prompts through the recurrent mixers: retention, wkv, mLSTM, the gated delta rule
        dict(name="retention_8b_2048", kind="retention", size="8b", tokens=2048, requests=1),
        dict(name="wkv_1b_1501", kind="wkv", size="1b", tokens=1501, requests=3),
        dict(name="mlstm_1b_2048", kind="mlstm", size="1b", tokens=2048, requests=1),
        dict(name="delta_8b_1024", kind="delta", size="8b", tokens=1024, requests=2),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["llama_decode", "llama_prompt", "llama_f32", "experts", "latent",
                       "retention", "wkv", "mlstm", "delta"])
    size = rng.choice(["1b", "8b"])
    if kind == "llama_decode":
        return dict(kind=kind, size=size, layers=4 if size == "8b" else 16,
                    batch=_log(rng, 1, 32), context=_log(rng, 100, 8000 if size == "8b" else 4000))
    if kind == "llama_prompt":
        tokens = _log(rng, 40, 2048)
        return dict(kind=kind, size=size, layers=4, tokens=tokens, requests=rng.randint(1, 4),
                    dtype="bfloat16")
    if kind == "llama_f32":
        return dict(kind="llama_prompt", size="1b", layers=2, tokens=_log(rng, 16, 600),
                    requests=rng.randint(1, 4), dtype="float32")
    if kind == "experts":
        return dict(kind=kind, size=size, unit=rng.choice(["gated", "relu_squared"]),
                    tokens=_log(rng, 1, 2048))
    return dict(kind=kind, size=size, tokens=_log(rng, 24, 2048), requests=rng.randint(1, 4))


def _lengths(case) -> list:
    """The requests' shares of the tokens: unequal, 1 : 2 : 3 ..., each at least one token."""
    n, total = case.get("requests", 1), case["tokens"]
    whole = n * (n + 1) // 2
    out = [max(1, total * (i + 1) // whole) for i in range(n)]
    out[-1] += total - sum(out)
    return out


# ------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + 17)


class _Draw:
    """Tensors in the order in which they are asked for, from one seed."""

    def __init__(self, seed, dtype):
        self.gen, self.dtype = _gen(seed), dtype

    def __call__(self, *shape, std=STD, mean=0.0, dtype=None):
        t = torch.empty(shape, dtype=dtype or self.dtype, device=DEV)
        return t.normal_(mean, std, generator=self.gen)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        t = torch.empty(shape, dtype=torch.float32, device=DEV)
        return t.uniform_(lo, hi, generator=self.gen)


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _llama_config(case) -> dict:
    return dict(LLAMA[case["size"]], architecture="llama_dense", n_layers=case["layers"],
                max_seq_len=CONTEXT, rope_theta=500000.0, norm_eps=EPS,
                dtype=case.get("dtype", "bfloat16"))


def _llama_tensors(case, seed):
    s, d = LLAMA[case["size"]], _Draw(seed, _dtype(case))
    w, q, kv, ff = (s["d_model"], s["n_heads"] * s["head_dim"], s["n_kv_heads"] * s["head_dim"],
                    s["intermediate_size"])
    t = {"embed.weight": d(s["vocab_size"], w)}
    for i in range(case["layers"]):
        b = f"blocks.{i}."
        t[b + "attn_norm.weight"] = d(w, std=0.1, mean=1.0)
        t[b + "attn.wq.weight"], t[b + "attn.wk.weight"] = d(q, w), d(kv, w)
        t[b + "attn.wv.weight"], t[b + "attn.wo.weight"] = d(kv, w), d(w, q)
        t[b + "mlp_norm.weight"] = d(w, std=0.1, mean=1.0)
        t[b + "mlp.w_gate.weight"], t[b + "mlp.w_up.weight"] = d(ff, w), d(ff, w)
        t[b + "mlp.w_down.weight"] = d(w, ff)
    t["final_norm.weight"] = d(w, std=0.1, mean=1.0)
    if not s["tie_embeddings"]:
        t["lm_head.weight"] = d(s["vocab_size"], w)
    return t, d


def _token_ids(case, seed, n) -> list:
    g = torch.Generator().manual_seed(7919 * int(seed) + 5)
    return torch.randint(0, LLAMA[case["size"]]["vocab_size"], (n,), generator=g).tolist()


def _decode_pool(case, d):
    """Keys and values of the contexts: [layers, 2, kv heads, pages, page, head size]."""
    s = LLAMA[case["size"]]
    pages = case["batch"] * (-(-(case["context"] + 1) // PAGE))
    return d(case["layers"], 2, s["n_kv_heads"], pages, PAGE, s["head_dim"], std=1.0)


def _experts_tensors(case, seed):
    s, d = SIZES[case["size"]], _Draw(seed, torch.bfloat16)
    w, ff, sh = s["width"], s["eff"], s["shared"]
    h = d(case["tokens"], w, std=1.0)
    t = {"router": d(s["experts"], w)}
    for i in range(s["experts"]):
        if case["unit"] == "gated":
            t[f"e{i}.gate"] = d(ff, w)
        t[f"e{i}.up"], t[f"e{i}.down"] = d(ff, w), d(w, ff)
    t["shared.gate"], t["shared.up"], t["shared.down"] = d(sh, w), d(sh, w), d(w, sh)
    if case["unit"] != "gated":
        t["router.b"] = d(s["experts"], std=0.5, dtype=torch.float32)
        t["shared.sg"] = d(1, w)
    return h, t


def _latent_tensors(case, seed):
    s, d = SIZES[case["size"]], _Draw(seed, torch.bfloat16)
    w, hd, r, rq = s["width"], s["heads"] * s["dim"], s["kv_rank"], s["q_rank"]
    h = d(case["tokens"], w, std=1.0)
    return h, {"dq": d(rq, w), "dq.norm": d(rq, std=0.1, mean=1.0), "uq": d(hd, rq, std=0.05),
               "dkv": d(r, w), "dkv.norm": d(r, std=0.1, mean=1.0), "uk": d(hd, r, std=0.08),
               "uv": d(hd, r, std=0.05), "o": d(w, hd)}


def _retention_decay(heads) -> list:
    return [1.0 - 2.0 ** (-5 - 3 * i / heads) for i in range(heads)]


def _retention_tensors(case, seed):
    s, d = SIZES[case["size"]], _Draw(seed, torch.bfloat16)
    w, c = s["width"], s["heads"] * s["dim"]
    h = d(case["tokens"], w, std=1.0)
    return h, {"q": d(c, w), "k": d(c, w), "v": d(2 * c, w), "g": d(2 * c, w), "o": d(w, 2 * c)}


def _wkv_tensors(case, seed):
    s, d = SIZES[case["size"]], _Draw(seed, torch.bfloat16)
    w = s["width"]
    h = d(case["tokens"], w, std=1.0)
    t = {f"mu.{n}": d.uniform(w).to(torch.bfloat16) for n in "rkvgw"}
    t.update({n: d(w, w) for n in "rkvg"})
    # decays of exp(-exp(w0)): from a few tokens to a few hundred
    t.update({"w1": d(64, w), "w2": d(w, 64), "w0": d.uniform(w, lo=-6.0, hi=-1.0).to(torch.bfloat16),
              "u": d(w // 64, 64, std=0.5), "norm": d(w, std=0.1, mean=1.0), "o": d(w, w)})
    return h, t


def _mlstm_tensors(case, seed):
    s, d = SIZES[case["size"]], _Draw(seed, torch.bfloat16)
    w, n, e, f = s["width"], s["mheads"], s["mdim"], s["mvdim"]
    h = d(case["tokens"], w, std=1.0)
    return h, {"q": d(n * e, w), "k": d(n * e, w), "v": d(n * f, w), "g": d(n * f, w),
               "o": d(w, n * f), "norm": d(n * f, std=0.1, mean=1.0), "i": d(n, w),
               "i.b": d(n, std=1.0), "f": d(n, w), "f.b": d(n, std=1.0, mean=3.0)}


def _delta_tensors(case, seed):
    s, d = SIZES[case["size"]], _Draw(seed, torch.bfloat16)
    w, n, e = s["width"], s["heads"], s["dim"]
    ck, cv = n // 2 * e, n * e
    h = d(case["tokens"], w, std=1.0)
    return h, {"q": d(ck, w), "q.conv": d(ck, 4, std=0.5), "k": d(ck, w), "k.conv": d(ck, 4, std=0.5),
               "v": d(cv, w), "v.conv": d(cv, 4, std=0.5), "b": d(n, w),
               "A_log": d.uniform(n, lo=0.0, hi=2.5).to(torch.bfloat16),
               "norm": d(e, std=0.1, mean=1.0), "a": d(n, w),
               "dt_bias": d.uniform(n, lo=-6.0, hi=-2.0).to(torch.bfloat16),
               "g": d(cv, w), "o": d(w, cv)}


_LAYER = {"experts": _experts_tensors, "latent": _latent_tensors, "retention": _retention_tensors,
          "wkv": _wkv_tensors, "mlstm": _mlstm_tensors, "delta": _delta_tensors}


def _part(case):
    s = SIZES[case["size"]]
    w, n, e = s["width"], s["heads"], s["dim"]
    kind = case["kind"]
    if kind == "experts":
        shared = SwiGLUFeedForward(w, s["shared"], names=("gate", "up", "down"))
        if case["unit"] == "gated":
            return RoutedExperts(w, s["experts"], s["top"], s["eff"], shared=shared, weigh="input")
        return RoutedExperts(w, s["experts"], s["top"], s["eff"], shared=shared, weigh="output",
                             score="logit", shared_gate=True, unit="relu_squared", router_bias=True)
    if kind == "latent":
        return LatentAttention(w, n, e, e, s["kv_rank"], s["q_rank"], e ** -0.5, EPS)
    if kind == "retention":
        return RetentionMixer(w, n, e, 2 * e, _retention_decay(n), EPS, PartialRotary(e, ROT_BASE))
    if kind == "wkv":
        return WkvMixer(w, w // 64, 64, 64, EPS)
    if kind == "mlstm":
        return MLstmMixer(w, s["mheads"], s["mdim"], s["mvdim"], GATE_CAP, EPS)
    return GatedDeltaMixer(w, n, n // 2, e, e, 4, EPS)


# ------------------------------------------------------------------------------------ program
def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("llama"):
        tensors, d = _llama_tensors(case, seed)
        dtype = _dtype(case)
        model = build_model(config_from_dict(_llama_config(case)))
        model.bind(tensors, Runtime(DEV, dtype))
        del tensors
        if kind == "llama_decode":
            n, ctx = case["batch"], case["context"]
            pool = _decode_pool(case, d)
            runner = ModelRunner(model, num_blocks=pool.shape[3], block_size=PAGE, max_requests=n)
            for i, handle in enumerate(runner.handles):
                handle.k_pool.copy_(pool[i, 0])
                handle.v_pool.copy_(pool[i, 1])
            for r in range(n):
                runner.cache.admit(r)
                runner.cache.reserve(r, ctx)
                runner.cache.commit(r, ctx)
            entries = [Entry(r, [t], [0]) for r, t in enumerate(_token_ids(case, seed, n))]
            return dict(kind=kind, runner=runner, entries=entries, context=ctx)
        lens = _lengths(case)
        ids = _token_ids(case, seed, sum(lens))
        runner = ModelRunner(model, num_blocks=sum(-(-n // PAGE) for n in lens), block_size=PAGE,
                             max_requests=len(lens))
        entries, at = [], 0
        for r, n in enumerate(lens):
            entries.append(Entry(r, ids[at:at + n], [n - 1]))
            at += n
        runner.reserve(entries)
        return dict(kind=kind, model=model, runner=runner, step=runner.builder.build(entries))
    h, tensors = _LAYER[kind](case, seed)
    part = _part(case)
    runtime = Runtime(DEV, torch.bfloat16)
    part.bind(tensors, runtime)
    del tensors
    if kind == "experts":
        return dict(kind=kind, part=part, h=h, ops=runtime.ops)
    lens = _lengths(case)
    cache = CacheManager([part.cache_spec()], num_blocks=sum(-(-n // PAGE) for n in lens),
                         block_size=PAGE, max_requests=len(lens), max_seq_len=CONTEXT, device=DEV,
                         kv_dtype=torch.bfloat16)
    builder = BatchBuilder(cache, DEV, 2, CONTEXT)
    for r, n in enumerate(lens):
        cache.admit(r)
        cache.reserve(r, n)
    step = builder.build([Entry(r, [0] * n) for r, n in enumerate(lens)])
    handle = cache.handles()[0]
    out = dict(kind=kind, part=part, h=h, ops=runtime.ops, cache=cache, builder=builder, step=step,
               handle=handle)
    s = SIZES[case["size"]]
    if kind == "mlstm":
        e, f = s["mdim"], s["mvdim"]
        out["state"] = handle.state[:, :, :e * f + e]
    elif kind == "delta":
        out["state"] = handle.state[:, :s["heads"] * s["dim"] * s["dim"]]
    elif kind != "latent":
        out["state"] = handle.state
    return out


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "llama_decode":
        runner = state["runner"]
        runner.reserve(state["entries"])
        logits = runner.step(state["entries"])
        # the next pass decodes the same token again
        for e in state["entries"]:
            runner.cache.truncate(e.owner, state["context"])
        return logits
    if kind == "llama_prompt":
        handles = state["runner"].handles
        logits = state["model"].forward(state["step"], handles)
        return {"logits": logits, "k": [c.k_pool for c in handles], "v": [c.v_pool for c in handles]}
    part, h = state["part"], state["h"]
    state["ops"].begin_step(h.shape[0])
    if kind == "experts":
        return part.forward(h, None)
    step, handle = state["step"], state["handle"]
    if kind == "latent":
        out = part.forward(h, step, handle)
        return {"out": out.float() if hasattr(out, "release") else out, "pool": handle.k_pool}
    handle.state.zero_()                     # the slots as new requests find them
    out = part.forward(h, step, handle)
    return {"out": out.float() if hasattr(out, "release") else out, "state": state["state"]}


# --------------------------------------------------------------------------------------- work
def work(case) -> dict:
    kind = case["kind"]
    if kind.startswith("llama"):
        s, size = LLAMA[case["size"]], 4 if case.get("dtype") == "float32" else 2
        w, q, kv, ff = (s["d_model"], s["n_heads"] * s["head_dim"],
                        s["n_kv_heads"] * s["head_dim"], s["intermediate_size"])
        layer = w * (2 * q + 2 * kv + 3 * ff)
        head = s["vocab_size"] * w
        n = case["layers"]
        if kind == "llama_decode":
            b, ctx = case["batch"], case["context"] + 1
            return {"bytes": size * (n * layer + head + n * b * ctx * 2 * kv) + 4 * b * s["vocab_size"],
                    "flops": 2 * b * (n * layer + head) + n * b * ctx * 4 * q}
        lens = _lengths(case)
        t, r = sum(lens), len(lens)
        return {"bytes": size * (n * layer + head + n * t * 2 * kv + t * w) + 4 * r * s["vocab_size"],
                "flops": 2 * t * n * layer + 2 * r * head + n * sum(2 * m * (m + 1) * q for m in lens)}
    s, t = SIZES[case["size"]], case["tokens"]
    w, n, e = s["width"], s["heads"], s["dim"]
    rows = 2 * 2 * t * w                                     # bfloat16 in and out
    if kind == "experts":
        mats = 3 if case["unit"] == "gated" else 2
        woken = s["experts"] * (1.0 - (1.0 - s["top"] / s["experts"]) ** t)
        shared = 3 * w * s["shared"]
        return {"bytes": rows + 2 * (woken * mats * w * s["eff"] + shared + s["experts"] * w),
                "flops": 2 * t * (s["top"] * mats * w * s["eff"] + shared + s["experts"] * w)}
    lens = _lengths(case)
    if kind == "latent":
        c, r, rq = n * e, s["kv_rank"], s["q_rank"]
        mats = w * (rq + r) + c * rq + 2 * c * r + w * c
        # scores and weighted sums over heads of e, two multiply-adds an entry and visible key
        return {"bytes": rows + 2 * mats + 2 * t * r,
                "flops": 2 * t * mats + sum(2 * m * (m + 1) * c for m in lens)}
    states = 2 * 4 * len(lens)                               # float32, in and out
    if kind == "retention":
        c = n * e
        return {"bytes": rows + 2 * w * 8 * c + states * n * e * 2 * e,
                "flops": 2 * t * w * 8 * c + t * n * 4 * e * 2 * e}
    if kind == "wkv":
        return {"bytes": rows + 2 * (5 * w * w + 2 * 64 * w) + states * (w * 64 + w),
                "flops": 2 * t * (5 * w * w + 2 * 64 * w) + t * w * 4 * 64}
    if kind == "mlstm":
        m, me, mf = s["mheads"], s["mdim"], s["mvdim"]
        mats = w * (2 * m * me + 3 * m * mf + 2 * m)
        return {"bytes": rows + 2 * mats + states * m * (me * mf + me), "flops": 2 * t * mats + t * m * 4 * me * mf}
    c = n * e
    mats = w * (2 * (c // 2) + 2 * c + 2 * n) + w * c
    return {"bytes": rows + 2 * mats + states * n * e * e, "flops": 2 * t * mats + t * n * 6 * e * e}


def tolerance(case):
    kind = case["kind"]
    if case.get("dtype") == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    if kind == "llama_decode":
        return {"rel": 2e-2, "max": 0.3}
    if kind == "llama_prompt":
        return {"rel": 2e-2, "max": 0.3}
    return {"rel": 1e-2, "max": 0.2}


# -------------------------------------------------------------------------------------- exact
def _f64(t):
    return t.double()


def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, base):
    """Halves of [T, H, e] turned by the positions 0 .. T-1 (or ``base`` = (theta, positions))."""
    theta, pos = base
    e = x.shape[-1]
    freq = torch.pow(torch.tensor(theta, dtype=torch.float64, device=DEV),
                     -2.0 * torch.arange(e // 2, dtype=torch.float64, device=DEV) / e)
    a = pos.double()[:, None] * freq
    c, s = a.cos()[:, None], a.sin()[:, None]
    x1, x2 = x[..., :e // 2], x[..., e // 2:]
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1)


def _causal(q, k, v, scale):
    """[T, H, e] queries over [T, G, e] keys and [T, G, f] values, head by head."""
    t, n, g = q.shape[0], q.shape[1], k.shape[1]
    hidden = torch.ones(t, t, dtype=torch.bool, device=DEV).triu(1)
    out = []
    for i in range(n):
        j = i // (n // g)
        s = (q[:, i] @ k[:, j].T) * scale
        out.append(torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ v[:, j])
    return torch.stack(out, 1)


def _pages_of(rows, lens):
    """Rows [T, ...] of the requests in pages of their own, the rest zero: [pages, PAGE, ...]."""
    out, at = [], 0
    for n in lens:
        p = rows.new_zeros((-(-n // PAGE) * PAGE,) + rows.shape[1:])
        p[:n] = rows[at:at + n]
        out.append(p.view(-1, PAGE, *rows.shape[1:]))
        at += n
    return torch.cat(out)


def _exact_llama(case, seed):
    tensors, d = _llama_tensors(case, seed)
    s = LLAMA[case["size"]]
    hd, nh, kv = s["head_dim"], s["n_heads"], s["n_kv_heads"]
    decode = case["kind"] == "llama_decode"
    pool = _decode_pool(case, d) if decode else None
    lens = [1] * case["batch"] if decode else _lengths(case)
    t = sum(lens)
    ids = torch.tensor(_token_ids(case, seed, t), device=DEV)
    x = _f64(tensors["embed.weight"][ids])
    starts = [sum(lens[:i]) for i in range(len(lens))]
    pos = (torch.full((t,), case["context"], device=DEV) if decode else
           torch.cat([torch.arange(n, device=DEV) for n in lens]))
    rope = (500000.0, pos)
    ks, vs = [], []
    for i in range(case["layers"]):
        w = {n[len(f"blocks.{i}."):-len(".weight")]: v for n, v in tensors.items()
             if n.startswith(f"blocks.{i}.")}
        h = _rms(x) * _f64(w["attn_norm"])
        q = _rotate((h @ _f64(w["attn.wq"]).T).view(t, nh, hd), rope)
        k = _rotate((h @ _f64(w["attn.wk"]).T).view(t, kv, hd), rope)
        v = (h @ _f64(w["attn.wv"]).T).view(t, kv, hd)
        o = torch.empty(t, nh, hd, dtype=torch.float64, device=DEV)
        if decode:
            n0 = -(-case["context"] // PAGE)
            for r in range(t):
                def past(which):
                    p = pool[i, which, :, r * n0:(r + 1) * n0]
                    return _f64(p.reshape(kv, n0 * PAGE, hd)[:, :case["context"]])
                kr = torch.cat([past(0), k[r][:, None]], 1)
                vr = torch.cat([past(1), v[r][:, None]], 1)
                a = torch.einsum("gqe,gke->gqk", q[r].view(kv, nh // kv, hd), kr) * hd ** -0.5
                o[r] = torch.einsum("gqk,gke->gqe", torch.softmax(a, -1), vr).reshape(nh, hd)
        else:
            for b, n in zip(starts, lens):
                o[b:b + n] = _causal(q[b:b + n], k[b:b + n], v[b:b + n], hd ** -0.5)
            ks.append(_pages_of(k, lens).permute(2, 0, 1, 3).contiguous())
            vs.append(_pages_of(v, lens).permute(2, 0, 1, 3).contiguous())
        x = x + o.reshape(t, nh * hd) @ _f64(w["attn.wo"]).T
        h = _rms(x) * _f64(w["mlp_norm"])
        x = x + (_silu(h @ _f64(w["mlp.w_gate"]).T) * (h @ _f64(w["mlp.w_up"]).T)) @ _f64(w["mlp.w_down"]).T
    last = torch.tensor([b + n - 1 for b, n in zip(starts, lens)], device=DEV)
    h = _rms(x[last]) * _f64(tensors["final_norm.weight"])
    head = tensors["embed.weight" if s["tie_embeddings"] else "lm_head.weight"]
    logits = h @ _f64(head).T
    return logits if decode else {"logits": logits, "k": ks, "v": vs}


def _exact_experts(case, seed):
    h, w = _experts_tensors(case, seed)
    s = SIZES[case["size"]]
    h = _f64(h)
    z = h @ _f64(w["router"]).T
    gated = case["unit"] == "gated"
    if gated:
        weight, idx = torch.sigmoid(z).topk(s["top"], -1)
    else:
        z = z + _f64(w["router.b"])
        best, idx = z.topk(s["top"], -1)
        weight = torch.softmax(best, -1)
    out = (_silu(h @ _f64(w["shared.gate"]).T) * (h @ _f64(w["shared.up"]).T)) @ _f64(w["shared.down"]).T
    if not gated:
        out = out * torch.sigmoid(h @ _f64(w["shared.sg"]).T)
    for i in range(s["experts"]):
        rows, place = (idx == i).nonzero(as_tuple=True)
        if not rows.numel():
            continue
        a, share = h[rows], weight[rows, place][:, None]
        up, down = _f64(w[f"e{i}.up"]), _f64(w[f"e{i}.down"])
        if gated:
            a = a * share
            y = (_silu(a @ _f64(w[f"e{i}.gate"]).T) * (a @ up.T)) @ down.T
        else:
            y = ((a @ up.T).clamp(min=0) ** 2) @ down.T * share
        out.index_add_(0, rows, y)
    return out


def _exact_latent(case, seed):
    h, w = _latent_tensors(case, seed)
    s = SIZES[case["size"]]
    n, e, t = s["heads"], s["dim"], case["tokens"]
    h = _f64(h)
    w = {k: _f64(v) for k, v in w.items()}
    q = (_rms(h @ w["dq"].T) * w["dq.norm"]) @ w["uq"].T
    c = _rms(h @ w["dkv"].T) * w["dkv.norm"]
    q, k, v = (a.view(t, n, e) for a in (q, c @ w["uk"].T, c @ w["uv"].T))
    lens, at, o = _lengths(case), 0, []
    for m in lens:
        o.append(_causal(q[at:at + m], k[at:at + m], v[at:at + m], e ** -0.5))
        at += m
    return {"out": torch.cat(o).reshape(t, n * e) @ w["o"].T, "pool": _pages_of(c, lens)[None]}


def _walk(case, one):
    """``one(first token, count)`` -> (outputs, state) of every request, put together."""
    outs, states, at = [], [], 0
    for n in _lengths(case):
        o, st = one(at, n)
        outs.append(o)
        states.append(st)
        at += n
    return torch.cat(outs), torch.stack(states)


def _exact_retention(case, seed):
    h, w = _retention_tensors(case, seed)
    s = SIZES[case["size"]]
    n, e, t = s["heads"], s["dim"], case["tokens"]
    f = 2 * e
    h = _f64(h)
    w = {k: _f64(v) for k, v in w.items()}
    q, k = ((h @ w[x].T).view(t, n, e) for x in "qk")
    v = (h @ w["v"].T).view(t, n, f)
    gamma = torch.tensor(_retention_decay(n), dtype=torch.float64, device=DEV).float().double()

    def one(at, m):
        pos = torch.arange(m, device=DEV)
        qr = _rotate(q[at:at + m], (ROT_BASE, pos))
        kr = _rotate(k[at:at + m], (ROT_BASE, pos)) * e ** -0.5
        vr = v[at:at + m]
        gap = (pos[:, None] - pos[None, :]).clamp(min=0).double()
        o = torch.empty(m, n, f, dtype=torch.float64, device=DEV)
        st = torch.empty(n, e, f, dtype=torch.float64, device=DEV)
        for i in range(n):
            a = (qr[:, i] @ kr[:, i].T) * (gamma[i] ** gap).tril()
            o[:, i] = a @ vr[:, i]
            st[i] = (kr[:, i] * (gamma[i] ** (m - 1 - pos).double())[:, None]).T @ vr[:, i]
        return o, st.reshape(-1)

    o, state = _walk(case, one)
    o = _rms(o).reshape(t, n * f) * _silu(h @ w["g"].T)
    return {"out": o @ w["o"].T, "state": state}


def _exact_wkv(case, seed):
    h, w = _wkv_tensors(case, seed)
    h = _f64(h)
    w = {k: _f64(v) for k, v in w.items()}
    t, d = h.shape
    n, e = d // 64, 64
    prev, at = torch.zeros_like(h), 0
    for m in _lengths(case):
        prev[at + 1:at + m] = h[at:at + m - 1]
        at += m
    mix = {x: h + (prev - h) * w[f"mu.{x}"] for x in "rkvgw"}
    r, k, v = ((mix[x] @ w[x].T).view(t, n, e) for x in "rkv")
    decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w["w1"].T) @ w["w2"].T + w["w0"])).view(t, n, e)
    u = w["u"]

    def one(at, m):
        st = torch.zeros(n, e, e, dtype=torch.float64, device=DEV)
        o = []
        for i in range(at, at + m):
            kv = k[i][:, :, None] * v[i][:, None, :]
            o.append(torch.einsum("hij,hi->hj", st + u[:, :, None] * kv, r[i]))
            st = decay[i][:, :, None] * st + kv
        return torch.stack(o), torch.cat([st.reshape(-1), h[at + m - 1]])

    o, state = _walk(case, one)
    o = _rms(o).reshape(t, d) * w["norm"] * _silu(mix["g"] @ w["g"].T)
    return {"out": o @ w["o"].T, "state": state}


def _exact_mlstm(case, seed):
    h, w = _mlstm_tensors(case, seed)
    s = SIZES[case["size"]]
    n, e, f, t = s["mheads"], s["mdim"], s["mvdim"], case["tokens"]
    h = _f64(h)
    w = {k: _f64(v) for k, v in w.items()}

    def cap(z):
        return GATE_CAP * torch.tanh(z / GATE_CAP)

    q = (h @ w["q"].T).view(t, n, e) * e ** -0.5
    k = (h @ w["k"].T).view(t, n, e)
    v = (h @ w["v"].T).view(t, n, f)
    ig = cap(h @ w["i"].T + w["i.b"])
    fg = torch.nn.functional.logsigmoid(cap(h @ w["f"].T + w["f.b"]))

    def one(at, m):
        c = torch.zeros(n, e, f, dtype=torch.float64, device=DEV)
        norm = torch.zeros(n, e, dtype=torch.float64, device=DEV)
        mx = torch.zeros(n, dtype=torch.float64, device=DEV)
        o = []
        for i in range(at, at + m):
            new = torch.maximum(fg[i] + mx, ig[i])
            keep, take = torch.exp(fg[i] + mx - new), torch.exp(ig[i] - new)
            mx = new
            c = keep[:, None, None] * c + (take[:, None] * k[i])[:, :, None] * v[i][:, None, :]
            norm = keep[:, None] * norm + take[:, None] * k[i]
            den = torch.maximum((norm * q[i]).sum(-1).abs(), torch.exp(-mx)) + 1e-6
            o.append(torch.einsum("hef,he->hf", c, q[i]) / den[:, None])
        return torch.stack(o), torch.cat([c.reshape(n, e * f), norm], 1)

    o, state = _walk(case, one)
    o = _rms(o).reshape(t, n * f) * w["norm"] * torch.sigmoid(h @ w["g"].T)
    return {"out": o @ w["o"].T, "state": state}


def _exact_delta(case, seed):
    h, w = _delta_tensors(case, seed)
    s = SIZES[case["size"]]
    n, e, t = s["heads"], s["dim"], case["tokens"]
    h = _f64(h)
    w = {k: _f64(v) for k, v in w.items()}
    rows = {x: h @ w[x].T for x in "qkv"}
    beta = torch.sigmoid(h @ w["b"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"]))

    def conv(x, at, m):
        u = torch.cat([torch.zeros(3, rows[x].shape[1], dtype=torch.float64, device=DEV),
                       rows[x][at:at + m]])
        return _silu(sum(u[j:j + m] * w[f"{x}.conv"][:, j] for j in range(4)))

    def one(at, m):
        q, k = (conv(x, at, m).view(m, n // 2, e) for x in "qk")
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * e ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        q, k = q.repeat_interleave(2, 1), k.repeat_interleave(2, 1)
        v = conv("v", at, m).view(m, n, e)
        st = torch.zeros(n, e, e, dtype=torch.float64, device=DEV)
        o = []
        for i in range(m):
            st = decay[at + i][:, None, None] * st
            u = beta[at + i][:, None] * (v[i] - torch.einsum("hef,he->hf", st, k[i]))
            st = st + k[i][:, :, None] * u[:, None, :]
            o.append(torch.einsum("hef,he->hf", st, q[i]))
        return torch.stack(o), st.transpose(1, 2).reshape(-1)

    o, state = _walk(case, one)
    o = (_rms(o) * w["norm"]).reshape(t, n * e) * _silu(h @ w["g"].T)
    return {"out": o @ w["o"].T, "state": state}


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("llama"):
        return _exact_llama(case, seed)
    return {"experts": _exact_experts, "latent": _exact_latent, "retention": _exact_retention,
            "wkv": _exact_wkv, "mlstm": _exact_mlstm, "delta": _exact_delta}[kind](case, seed)
