"""The work that programs built on this framework give it, as cases that can be timed and compared.

Each case is one public entry point at sizes from the CLI presets, the benchmark model or the tests: the layers of a
training step (attention, feed-forward, mixture of experts, norm, language-model head), one generation step with a KV
cache, and a whole captured training step. The layers run forward and backward with their parameters in the flat arena
that ``engine.prepare_training`` sets up, as a training step runs them. ``exact`` restates each path in 64 bits.
"""
import math

import torch
import torch.nn.functional as F

from nanopysche_b200.engine import GraphedTrainStep, prepare_training
from nanopysche_b200.fp8.training import FP8Config, apply_fp8
from nanopysche_b200.models.attention import Attention
from nanopysche_b200.models.feed_forward import FeedForward
from nanopysche_b200.models.moe import MoEBase
from nanopysche_b200.models.norm import RMSNorm
from nanopysche_b200.models.transformer import Transformer
from nanopysche_b200.ops.gemm import linear
from nanopysche_b200.ops.xent import cross_entropy

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
ROPE_BASE = 10000.0
LR, WD, BETAS, EPS, CLIP = 3e-4, 0.1, (0.9, 0.95), 1e-8, 1.0   # the CLI's optimizer settings
GRAPH_WARMUP = 3   # eager steps that GraphedTrainStep takes before it captures


def listed():
    return [
        # a layer of the 125m preset on a short context: heads of 64, small matrices, launches count
        dict(name="attention_125m", kind="attention", batch=4, seq=1024, d_model=768, heads=12, kv_heads=12, head_dim=64,
             qk_norm=False, causal=True),
        # the attention layer of the benchmark model (16 query / 8 KV heads of 128) at its batch
        dict(name="attention_gqa", kind="attention", batch=2, seq=2048, d_model=2048, heads=16, kv_heads=8, head_dim=128,
             qk_norm=False, causal=True),
        # the same layer on a long context: the score products dominate
        dict(name="attention_long", kind="attention", batch=1, seq=8192, d_model=2048, heads=16, kv_heads=8, head_dim=128,
             qk_norm=False, causal=True),
        # an odd sequence length, per-head norms, no mask (a bidirectional encoder or a prefix)
        dict(name="attention_ragged", kind="attention", batch=3, seq=777, d_model=2048, heads=16, kv_heads=8,
             head_dim=128, qk_norm=True, causal=False),
        # one generation step of the benchmark model's attention layer for a small batch with a filled cache
        dict(name="attention_decode", kind="decode", batch=8, past=2047, d_model=2048, heads=16, kv_heads=8,
             head_dim=128),
        # the feed-forward of the 1b presets at the benchmark's 4096 tokens
        dict(name="feed_forward_1b", kind="feed_forward", tokens=4096, d_model=2048, hidden=5632, act="silu", fp8="none"),
        # the same with e4m3 forward operands, the fp8 training option
        dict(name="feed_forward_mxfp8", kind="feed_forward", tokens=4096, d_model=2048, hidden=5632, act="silu",
             fp8="mxfp8"),
        # the mixture-of-experts layer of the benchmark model
        dict(name="moe_1b", kind="moe", tokens=4096, d_model=2048, hidden=2816, experts=8, top_k=2, capacity=1.25),
        # a small expert layer without a capacity limit, where launches and small kernels count
        dict(name="moe_small", kind="moe", tokens=512, d_model=768, hidden=2048, experts=8, top_k=2, capacity=0.0),
        # norm with the residual add in front, as every block runs it twice
        dict(name="norm_residual", kind="norm", tokens=4096, d_model=2048),
        # language-model head and loss of the benchmark model
        dict(name="head_loss", kind="head", tokens=4096, d_model=2048, vocab=32000),
        # a whole training step (forward, backward, clip, AdamW) replayed as one graph: four layers at the 350m widths
        dict(name="train_step", kind="step", batch=2, seq=1024, d_model=1024, layers=4, heads=16, kv_heads=16,
             head_dim=64, hidden=2816, vocab=32000),
    ]


def _log(rng, lo, hi, multiple=1):
    """A size spread over the logarithm of its range, rounded to ``multiple``."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    """One more case of these ranges, no costlier than the largest listed one."""
    top = [work(c) for c in listed()]
    while True:
        c = _draw(rng)
        w = work(c)
        if all(w[k] <= max(t[k] for t in top) for k in ("bytes", "flops")):
            return c


def _draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "decode", "feed_forward", "moe", "moe", "norm", "head",
                       "step"])
    if kind in ("attention", "decode"):
        d_model, heads, kv_heads, hd = rng.choice([(768, 12, 12, 64), (1024, 16, 16, 64), (2048, 32, 32, 64),
                                                   (2048, 16, 8, 128), (4096, 32, 8, 128)])
        if kind == "decode":
            return dict(kind=kind, batch=_log(rng, 1, 32), past=_log(rng, 64, 4096), d_model=d_model, heads=heads,
                        kv_heads=kv_heads, head_dim=hd)
        seq = _log(rng, 128, 6000)
        batch = max(1, min(8, _log(rng, 1, max(1.1, 6000 * 2048 / (seq * d_model)))))
        return dict(kind=kind, batch=batch, seq=seq, d_model=d_model, heads=heads, kv_heads=kv_heads, head_dim=hd,
                    qk_norm=hd == 128 and rng.random() < 0.3, causal=rng.random() < 0.8)
    if kind == "feed_forward":
        d_model, hidden = rng.choice([(768, 2048), (1024, 2816), (2048, 5632)])
        return dict(kind=kind, tokens=_log(rng, 128, 8192), d_model=d_model, hidden=hidden,
                    act=rng.choice(["silu", "silu", "gelu_tanh"]), fp8=rng.choice(["none", "none", "mxfp8"]))
    if kind == "moe":
        d_model, hidden = rng.choice([(768, 2048), (1024, 2816), (2048, 2816)])
        return dict(kind=kind, tokens=_log(rng, 256, 4096, 8), d_model=d_model, hidden=hidden,
                    experts=rng.choice([4, 8, 16]), top_k=rng.choice([1, 2, 2, 4]),
                    capacity=rng.choice([0.0, 1.25, 1.5, 2.0]))
    if kind == "norm":
        return dict(kind=kind, tokens=_log(rng, 64, 16384), d_model=rng.choice([768, 1024, 2048, 4096]))
    if kind == "head":
        return dict(kind=kind, tokens=_log(rng, 256, 4096), d_model=rng.choice([768, 1024, 2048]),
                    vocab=rng.choice([32000, 32000, 50264]))
    d_model, heads, hidden = rng.choice([(768, 12, 2048), (1024, 16, 2816)])
    return dict(kind=kind, batch=rng.choice([1, 2, 4]), seq=_log(rng, 128, 1024), d_model=d_model,
                layers=rng.choice([1, 2, 4]), heads=heads, kv_heads=heads, head_dim=64, hidden=hidden, vocab=32000)


# ---------------------------------------------------------------------------------------------------------- inputs
class _Gen:
    """Seeded normal tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + 17)

    def __call__(self, *shape, std=1.0, dtype=BF16):
        return (torch.randn(*shape, device="cuda", dtype=F32, generator=self.g) * std).to(dtype)

    def ints(self, high, *shape):
        return torch.randint(0, high, shape, device="cuda", generator=self.g)


def _fill(module, gen, skip=()):
    """Normal(0, 0.02) matrices and norm weights near one, as a model some way into training has them."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.dim() >= 2:
                p.copy_(gen(*p.shape, std=0.02, dtype=F32))
            elif name.endswith("norm.weight") or name == "weight":
                p.copy_(1.0 + gen(*p.shape, std=0.1, dtype=F32))
            elif name not in skip:
                p.copy_(gen(*p.shape, std=0.02, dtype=F32))
    return module


def _attention(c, gen):
    m = Attention(d_model=c["d_model"], n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=c["head_dim"],
                  rope_base=ROPE_BASE, max_seq_len=c.get("seq", c.get("past", 0) + 1), qk_norm=c.get("qk_norm", False),
                  dtype=BF16, device="cuda")
    return _fill(m, gen)


def _build(c, seed):
    """The module and the inputs of a case, in a fixed order of draws: ``prepare`` and ``exact`` see the same values."""
    g, kind, D = _Gen(seed), c["kind"], c["d_model"]
    if kind == "attention":
        B, S = c["batch"], c["seq"]
        return dict(m=_attention(c, g), x=g(B, S, D), dy=g(B, S, D, std=0.01))
    if kind == "decode":
        kv = (c["batch"], c["past"], c["kv_heads"], c["head_dim"])
        return dict(m=_attention(c, g), x=g(c["batch"], 1, D), k=g(*kv), v=g(*kv))
    if kind == "feed_forward":
        m = FeedForward(d_model=D, hidden_size=c["hidden"], activation=c["act"], dtype=BF16, device="cuda")
        return dict(m=_fill(m, g), x=g(1, c["tokens"], D), dy=g(1, c["tokens"], D, std=0.01))
    if kind == "moe":
        m = MoEBase(d_model=D, hidden_size=c["hidden"], num_experts=c["experts"], top_k=c["top_k"],
                    capacity_factor=c["capacity"] or None, dtype=BF16, device="cuda")
        return dict(m=_fill(m, g), x=g(1, c["tokens"], D), dy=g(1, c["tokens"], D, std=0.01))
    if kind == "norm":
        T = c["tokens"]
        return dict(m=_fill(RMSNorm(D, device="cuda"), g), x=g(1, T, D), res=g(1, T, D, std=2.0),
                    dy=g(1, T, D, std=0.01), dh=g(1, T, D, std=0.01))
    if kind == "head":
        m = torch.nn.Linear(D, c["vocab"], bias=False, dtype=BF16, device="cuda")
        labels = g.ints(c["vocab"], c["tokens"])
        labels[::17] = -100   # padding and the last position of a sequence carry no label
        return dict(m=_fill(m, g), x=g(c["tokens"], D), labels=labels)
    m = Transformer(d_model=D, vocab_size=c["vocab"], n_layers=c["layers"], dtype=BF16, init_device="cuda",
                    block=dict(n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=c["head_dim"], rope_base=ROPE_BASE,
                               max_seq_len=c["seq"], qk_norm=False, ffn_hidden=c["hidden"]))
    return dict(m=_fill(m, g), ids=g.ints(c["vocab"], c["batch"], c["seq"]))


def prepare(case, seed):
    s = _build(case, seed)
    kind = case["kind"]
    s["kind"], s["causal"] = kind, case.get("causal", True)
    if kind == "decode":
        s["start"] = case["past"]
        s["m"].requires_grad_(False)
        return s
    if case.get("fp8", "none") != "none":
        apply_fp8(s["m"], FP8Config(enabled=True, recipe_name=case["fp8"]))
    s["opt"], s["arena"] = prepare_training(s["m"], tokens_per_rank=case.get("tokens"), lr=LR, betas=BETAS, eps=EPS,
                                            weight_decay=WD, max_grad_norm=CLIP)
    if kind == "step":
        s["step"] = GraphedTrainStep(s["m"], s["opt"], s["ids"], warmup=GRAPH_WARMUP).capture()
    for k in ("x", "res"):
        if k in s:
            s[k].requires_grad_(True)
    return s


# --------------------------------------------------------------------------------------------------------- one pass
def run(s):
    kind, m = s["kind"], s["m"]
    if kind == "decode":
        with torch.no_grad():
            y, (k, v) = m(s["x"], kv_cache=(s["k"], s["v"]), start_pos=s["start"], return_kv=True)
        return dict(y=y, k=k, v=v)
    if kind == "step":
        loss = s["step"].step(s["ids"])
        return dict(loss=loss, weights={n: p.detach() for n, p in m.named_parameters()})
    x = s["x"]
    x.grad = None
    if kind == "attention":
        y = m(x, causal=s["causal"])
        y.backward(s["dy"])
        out = dict(y=y)
    elif kind == "feed_forward":
        y = m(x)
        y.backward(s["dy"])
        out = dict(y=y)
    elif kind == "moe":
        y = m(x)
        aux = m.aux_loss
        torch.autograd.backward([y, aux], [s["dy"], torch.ones_like(aux)])
        out = dict(y=y, aux=aux.detach())
    elif kind == "norm":
        s["res"].grad = None
        y, h = m(x, residual=s["res"])
        torch.autograd.backward([y, h], [s["dy"], s["dh"]])
        out = dict(y=y, h=h, dres=s["res"].grad)
    else:
        logits = linear(x, m.weight)
        loss = cross_entropy(logits, s["labels"])
        loss.backward()
        out = dict(loss=loss.detach(), logits=logits)
    out["dx"] = x.grad
    out["grads"] = {n: g.view(g.shape) for n, g in s["arena"].named_main_grads()}
    s["opt"].zero_grad()   # the next pass overwrites the gradient buffers; nothing is cleared here
    return {k: v.detach() if isinstance(v, torch.Tensor) else v for k, v in out.items()}


# -------------------------------------------------------------------------------------------------------------- work
def work(case):
    c, kind, D = case, case["kind"], case["d_model"]
    if kind in ("attention", "decode"):
        q, kv = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
        par = D * (2 * q + 2 * kv)
        if kind == "decode":
            n = c["batch"] * (c["past"] + 1)
            return dict(bytes=2.0 * par + 2 * 2 * 2.0 * n * kv + 4.0 * c["batch"] * D,
                        flops=2.0 * c["batch"] * par + 4.0 * n * q)
        T = c["batch"] * c["seq"]
        score = 2.0 * T * c["seq"] * q * (0.5 if c["causal"] else 1.0)   # one score-sized product
        return dict(bytes=2.0 * 4 * T * D + (2.0 + 4.0) * par, flops=6.0 * T * par + 7 * score)
    if kind == "feed_forward":
        par = 3.0 * D * c["hidden"]
        return dict(bytes=2.0 * 4 * c["tokens"] * D + 6.0 * par, flops=6.0 * c["tokens"] * par)
    if kind == "moe":
        par = 3.0 * c["experts"] * D * c["hidden"]
        rows = c["tokens"] * c["top_k"]
        return dict(bytes=2.0 * 4 * c["tokens"] * D + 6.0 * par, flops=18.0 * rows * D * c["hidden"])
    if kind == "norm":
        return dict(bytes=2.0 * 8 * c["tokens"] * D, flops=12.0 * c["tokens"] * D)
    if kind == "head":
        par = float(D) * c["vocab"]
        return dict(bytes=2.0 * 2 * c["tokens"] * D + 2.0 * c["tokens"] * c["vocab"] + 6.0 * par,
                    flops=6.0 * c["tokens"] * par)
    q, kv, T = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c["batch"] * c["seq"]
    mat = c["layers"] * (D * (2 * q + 2 * kv) + 3 * D * c["hidden"]) + D * c["vocab"]
    score = 2.0 * T * c["seq"] * q * 0.5 * c["layers"]
    return dict(bytes=26.0 * (mat + D * c["vocab"]), flops=6.0 * T * mat + 7 * score)


def tolerance(case):
    """About four times the distance from ``exact`` that was measured on the cases above (bf16 results and bf16
    intermediates; the worst output of each kind), and the largest single deviation such results show."""
    kind = case["kind"]
    if kind == "norm":
        return {"rel": 8e-3, "max": 0.1}
    if kind == "head":
        return {"rel": 7e-3, "max": 0.1}
    if kind == "step":
        return {"rel": 1.2e-2, "max": 0.5}
    if kind == "decode":
        return {"rel": 1.4e-2, "max": 0.2}
    if kind == "moe":
        # a token whose two best experts tie to the last bits of the logits may go to the other one: whole rows differ
        return {"rel": 1.8e-2, "max": 0.99}
    if kind == "feed_forward":
        # e4m3 operands: a last-bit change of an activation can move it to the next e4m3 value, a step of 1/16
        return {"rel": 1.4e-2, "max": 0.3} if case["fp8"] == "none" else {"rel": 3e-2, "max": 0.9}
    return {"rel": 2.5e-2 if case["qk_norm"] else 2e-2, "max": 0.4}


# ------------------------------------------------------------------------------------------------- the path in 64 bits
def _d(t):
    return t.detach().to(F64)


def _rope(x, start):
    """Half-split rotation of ``x [B, S, H, hd]`` at positions ``start ...``."""
    S, hd = x.shape[1], x.shape[3]
    inv = ROPE_BASE ** (-torch.arange(0, hd, 2, device=x.device, dtype=F64) / hd)
    ang = torch.outer(torch.arange(start, start + S, device=x.device, dtype=F64), inv)
    c, s = ang.cos()[None, :, None], ang.sin()[None, :, None]
    a, b = x[..., : hd // 2], x[..., hd // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _softmax_attention(q, k, v, causal):
    rep = q.shape[2] // k.shape[2]
    out = []
    for b in range(q.shape[0]):
        heads = []
        for h in range(q.shape[2]):
            s = q[b, :, h] @ k[b, :, h // rep].t() / math.sqrt(q.shape[3])
            if causal:
                vis = torch.ones(s.shape, device=s.device, dtype=torch.bool).tril(k.shape[1] - q.shape[1])
                s = s.masked_fill(~vis, float("-inf"))
            heads.append(s.softmax(-1) @ v[b, :, h // rep])
        out.append(torch.stack(heads, 1))
    return torch.stack(out)


def _attention64(w, x, c, causal, cache=None, start=0):
    B, S, hd = x.shape[0], x.shape[1], c["head_dim"]
    q, k, v = (F.linear(x, w[n + ".weight"]).view(B, S, -1, hd) for n in ("w_q", "w_k", "w_v"))
    if c.get("qk_norm"):
        q = F.layer_norm(q, (hd,), w["q_norm.weight"], w["q_norm.bias"], 1e-5)
        k = F.layer_norm(k, (hd,), w["k_norm.weight"], w["k_norm.bias"], 1e-5)
    q, k = _rope(q, start), _rope(k, start)
    if cache is not None:
        k, v = torch.cat([cache[0], k], 1), torch.cat([cache[1], v], 1)
    return F.linear(_softmax_attention(q, k, v, causal).reshape(B, S, -1), w["w_out.weight"]), k, v


def _feed_forward64(w, x, act):
    g = F.linear(x, w["w1.weight"])
    a = F.silu(g) if act == "silu" else F.gelu(g, approximate="tanh")
    return F.linear(a * F.linear(x, w["w3.weight"]), w["w2.weight"])


def _moe64(w, x, c):
    T, E, K, H = c["tokens"], c["experts"], c["top_k"], c["hidden"]
    x2 = x.reshape(T, -1)
    logits = F.linear(x2, w["router.gate.weight"], w["router.gate.bias"])
    top, idx = logits.topk(K, -1)
    gate = top.softmax(-1)
    hit = torch.zeros(T, E, device=x.device, dtype=F64).scatter_(1, idx, 1.0)
    aux = E * (hit.mean(0) * logits.softmax(-1).mean(0)).sum()
    keep = torch.ones(T, device=x.device, dtype=torch.bool)
    if c["capacity"]:
        keep = ~((hit > 0) & (hit.cumsum(0) > int(c["capacity"] * T / E))).any(1)
    y = torch.zeros_like(x2)
    for e in range(E):
        t, k = ((idx == e) & keep[:, None]).nonzero(as_tuple=True)
        r = slice(e * H, (e + 1) * H)
        xe = x2[t]
        ye = (F.silu(xe @ w["w1"][r].t()) * (xe @ w["w3"][r].t())) @ w["w2"][r]
        y = y.index_add(0, t, ye * gate[t, k][:, None])
    return y.view(x.shape), aux


def _norm64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * w


def _step64(s, c):
    """The warm-up steps of the captured step and one more, all on the same batch."""
    w = {n: _d(p).requires_grad_(True) for n, p in s["m"].named_parameters()}
    m1 = {n: torch.zeros_like(p) for n, p in w.items()}
    m2 = {n: torch.zeros_like(p) for n, p in w.items()}
    ids = s["ids"]
    tgt = torch.full_like(ids, -100)
    tgt[:, :-1] = ids[:, 1:]
    for t in range(1, GRAPH_WARMUP + 2):
        x = F.embedding(ids, w["embeddings.weight"])
        for i in range(c["layers"]):
            def sub(part):
                pre = "blocks.%d.%s." % (i, part)
                return {n[len(pre):]: p for n, p in w.items() if n.startswith(pre)}
            x = x + _attention64(sub("attention"), _norm64(x, sub("attention_norm")["weight"]), c, True)[0]
            x = x + _feed_forward64(sub("feed_forward"), _norm64(x, sub("feed_forward_norm")["weight"]), "silu")
        loss = F.cross_entropy(F.linear(x, w["lm_head.weight"]).flatten(0, 1), tgt.reshape(-1), ignore_index=-100)
        grads = torch.autograd.grad(loss, list(w.values()))
        scale = min(1.0, CLIP / (float(sum(g.pow(2).sum() for g in grads)) ** 0.5 + 1e-6))
        with torch.no_grad():
            for (n, p), g in zip(w.items(), grads):
                g = g * scale
                m1[n].mul_(BETAS[0]).add_(g, alpha=1 - BETAS[0])
                m2[n].mul_(BETAS[1]).addcmul_(g, g, value=1 - BETAS[1])
                decay = 0.0 if ("norm" in n or "emb" in n or p.dim() < 2) else WD
                p.mul_(1 - LR * decay)
                p.sub_(LR * (m1[n] / (1 - BETAS[0] ** t)) / ((m2[n] / (1 - BETAS[1] ** t)).sqrt() + EPS))
    return dict(loss=loss.detach(), weights={n: p.detach() for n, p in w.items()})


def exact(case, seed):
    c, s = case, _build(case, seed)
    kind = c["kind"]
    if kind == "step":
        return _step64(s, c)
    w = {n: _d(p).requires_grad_(True) for n, p in s["m"].named_parameters()}
    x = _d(s["x"])
    if kind == "decode":
        with torch.no_grad():
            y, k, v = _attention64(w, x, c, True, (_d(s["k"]), _d(s["v"])), c["past"])
        return dict(y=y, k=k, v=v)
    x.requires_grad_(True)
    leaves = [x, *w.values()]
    if kind == "attention":
        y = _attention64(w, x, c, c["causal"])[0]
        out, top, seeds = dict(y=y), [y], [_d(s["dy"])]
    elif kind == "feed_forward":
        y = _feed_forward64(w, x, c["act"])
        out, top, seeds = dict(y=y), [y], [_d(s["dy"])]
    elif kind == "moe":
        y, aux = _moe64(w, x, c)
        out, top, seeds = dict(y=y, aux=aux), [y, aux], [_d(s["dy"]), torch.ones_like(aux)]
    elif kind == "norm":
        h = x + _d(s["res"])
        y = _norm64(h, w["weight"])
        out, top, seeds = dict(y=y, h=h), [y, h], [_d(s["dy"]), _d(s["dh"])]
    else:
        logits = F.linear(x, w["weight"])
        loss = F.cross_entropy(logits, s["labels"], ignore_index=-100)
        out, top, seeds = dict(loss=loss, logits=logits), [loss], [torch.ones_like(loss)]
    grads = torch.autograd.grad(top, leaves, seeds)
    out["dx"] = grads[0]
    if kind == "norm":
        out["dres"] = grads[0]
    out["grads"] = dict(zip(w, grads[1:]))
    return {k: v.detach() if isinstance(v, torch.Tensor) else v for k, v in out.items()}
