"""Kernels in a graph start while the kernel in front of them drains (programmatic launch). Each reads what that one writes, so
a load that does not wait shows as a value of the replay before (GPU only)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

T, D, V, E, K = 515, 256, 1000, 8, 2


def _state():
    g = torch.Generator(device="cuda").manual_seed(5)

    def r(*s, std=1.0, dtype=torch.bfloat16):
        return (torch.randn(*s, device="cuda", generator=g) * std).to(dtype)

    from nanopysche_b200.ops.rope import rope_tables

    s = dict(x=r(1, T, D), res=r(1, T, D), labels=torch.randint(0, V, (T,), device="cuda", generator=g), norm=r(D, dtype=torch.float32),
             wqkv=r(3 * D, D, std=0.06), w13=r(2 * 512, D, std=0.06), w2=r(D, 512, std=0.05), head=r(V, D, std=0.06),
             gate=r(E, D, std=0.1, dtype=torch.float32), bias=r(E, dtype=torch.float32))
    s["rope"] = rope_tables(T, 64, device="cuda")
    s["p"], s["m"], s["v"] = r(V * D, dtype=torch.float32), *(torch.zeros(V * D, device="cuda") for _ in range(2))
    return s


def _chain(s):
    """A token's way through the layers, the loss and its gradient, one optimizer step: every kernel's input is the output of
    the one before. All sums are in a fixed order."""
    from nanopysche_b200.ops import _lib
    from nanopysche_b200.ops.attention import attention, attention_append
    from nanopysche_b200.ops.gemm import feed_forward_glu, linear
    from nanopysche_b200.ops.moe import _Router
    from nanopysche_b200.ops.norm import rms_norm
    from nanopysche_b200.ops.rope import qkv_rope
    from nanopysche_b200.ops.xent import cross_entropy

    with torch.no_grad():
        y, h = rms_norm(s["x"], s["norm"], 1e-6, s["res"])
        q, k, v = qkv_rope(linear(y, s["wqkv"]), *s["rope"], 4, 4, 64)
        a = attention(q, k, v).reshape(1, T, D)
        one, kc, vc = attention_append(q[:, -1:], k, v, k[:, -1:], v[:, -1:])      # a generation step, then its few-row linear
        few = linear(one.reshape(1, D), s["head"])
        f = feed_forward_glu(a, s["w13"], s["w2"])
        w, idx, _, counts = _Router.apply(f.view(T, D), s["gate"], s["bias"], None, K, 0, 0.0)
        plan = [torch.empty(n, device="cuda", dtype=torch.int32) for n in ((T, K), (T,), (E,), (E,), (1,), (2,))]
        _lib.call("capacity_plan", idx, T, E, K, 140, *plan, 2, None)
        f.mul_(plan[1].view(1, T, 1))
    logits = linear(f.view(T, D), s["head"]).detach().requires_grad_(True)
    loss = cross_entropy(logits, s["labels"])
    (dl,) = torch.autograd.grad(loss, logits)
    with torch.no_grad():
        gw = torch.empty(V, D, device="cuda")
        from nanopysche_b200.ops.gemm import gemm

        gemm(dl, f.view(T, D), a_mn=True, b_mn=True, out=gw)
        part, coef = torch.empty(_lib.lib().np_sumsq_parts(), device="cuda"), torch.empty(2, device="cuda")
        _lib.call("sumsq", gw, _lib.LL(gw.numel()), part)
        _lib.call("clip_coef", part, part.numel(), None, 0.1, coef)
        p, m, v2 = (s[n].clone() for n in ("p", "m", "v"))
        _lib.call("adamw", p, gw, m, v2, None, _lib.LL(p.numel()), 1e-3, 0.9, 0.95, 1e-8, 0.1, 1, coef, None)
    return [y, h, a, one, kc, vc, few, w, idx, counts, *plan, f, logits.detach(), loss.detach(), dl, gw, coef, p, m, v2]


def test_replays_see_this_replays_values():
    s = _state()
    g = torch.Generator(device="cuda").manual_seed(6)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            _chain(s)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _chain(s)
    for i in range(60):
        s["x"].copy_(torch.randn(1, T, D, device="cuda", generator=g) * (1 + i % 3))
        s["labels"].copy_(torch.randint(0, V, (T,), device="cuda", generator=g))
        want = [t.clone() for t in _chain(s)]
        for t in out:                       # whatever the last replay left is gone
            t.zero_()
        graph.replay()
        bad = [j for j, (a, b) in enumerate(zip(out, want)) if not torch.equal(a, b)]
        assert not bad, (i, bad)
