"""Row-wise and token-wise kernels at the edges of their blocking, against fp64 PyTorch (GPU only). Tolerances: one rounding
of the result to bf16 (2-norm 0.0017) plus fp32 sums, doubled; fp32 results 1e-5."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b.double()).norm() / (b.double().norm() + 1e-30)).item()


# rows off the two- and four-row batches and fewer than one, both sides of the switch between them (592 rows) and of the one
# to a CTA per row (2048 columns), several groups per CTA (above 1184 rows of at most 1024 columns), columns off a warp's 256
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 768), (5, 2048), (1023, 1032), (1187, 4096), (2600, 768), (9, 6144),
                                       (297, 2048), (591, 264), (593, 2040), (300, 2056), (700, 4104),
                                       (1184, 1024), (1185, 1024), (2403, 264), (3001, 8), (2371, 520), (9601, 768)])
@pytest.mark.parametrize("res", [False, True])
def test_rmsnorm_rows(rows, cols, res):
    from nanopysche_b200.ops.norm import rms_norm

    torch.manual_seed(rows)
    x, r, dy, dh = (torch.randn(rows, cols, device="cuda").bfloat16() for _ in range(4))
    w = (torch.rand(cols, device="cuda") + 0.5).requires_grad_(True)
    xa, ra = x.clone().requires_grad_(True), r.clone().requires_grad_(True)
    out = rms_norm(xa, w, 1e-6, ra if res else None)
    y, h = out if res else (out, None)
    torch.autograd.backward([y, h] if res else [y], [dy, dh] if res else [dy])
    x64, w64 = x.double().requires_grad_(True), w.detach().double().requires_grad_(True)
    h64 = x64 + r.double() if res else x64
    y64 = h64 * torch.rsqrt(h64.pow(2).mean(-1, keepdim=True) + 1e-6) * w64
    torch.autograd.backward([y64, h64] if res else [y64], [dy.double(), dh.double()] if res else [dy.double()])
    assert rel(y, y64) < 4e-3 and rel(xa.grad, x64.grad) < 5e-3 and rel(w.grad, w64.grad) < 5e-3


# rows shorter than a vector per thread, a tail off the vectors, a row stride above the row's length
@pytest.mark.parametrize("rows,V", [(3, 9), (70, 1003), (5, 16384), (33, 32000), (9, 50264), (2, 70003)])
def test_cross_entropy_rows(rows, V):
    from nanopysche_b200.ops.xent import cross_entropy

    torch.manual_seed(V)
    ld = (V + 7) // 8 * 8
    base = (torch.randn(rows, ld, device="cuda") * 3).bfloat16()
    logits = base[:, :V].detach().requires_grad_(True)
    labels = torch.randint(0, V, (rows,), device="cuda")
    labels[0] = -100
    labels[-1] = V - 1
    loss = cross_entropy(logits, labels)
    loss.backward()
    l64 = logits.detach().double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(l64, labels, ignore_index=-100)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 1e-5 * abs(ref.item()) and rel(logits.grad, l64.grad) < 4e-3


# The sum of a row is formed in one order against the row's maximum: bits of lse, taken from the two-pass kernel. One large entry per
# row keeps the logarithm small, so that the last bits of the sum show.
LSE_BITS = {1003: [1058881404, 1058961473, 1058751203, 1059190132, 1059210456, 1059747382],
            32000: [1079399911, 1079429039, 1079425302, 1079415901, 1079391680, 1079416142],
            50264: [1081257709, 1081275162, 1081247448, 1081250681, 1081248575, 1081272020]}


@pytest.mark.parametrize("V", LSE_BITS)
def test_cross_entropy_order_of_the_sum(V):
    from nanopysche_b200.ops.xent import _rows_fwd

    r, c = torch.arange(6), torch.arange((V + 7) // 8 * 8)
    x = -5 - ((r[:, None] * 7919 + c * 104729 + c * c % 1543) % 2003).float() / 256
    x[r, r * 17 + V // 2] = 0.0
    _, lse = _rows_fwd(x.bfloat16().cuda()[:, :V], torch.zeros(6, dtype=torch.long, device="cuda"), -100)
    assert lse.view(torch.int32).tolist() == LSE_BITS[V]


# masked vocabulary entries (-inf): single ones, a thread's whole share, all but one; +inf, NaN and a row of -inf give NaN
@pytest.mark.parametrize("V", [7, 264, 8200, 32000])
def test_cross_entropy_infinities(V):
    from nanopysche_b200.ops.xent import _rows_fwd

    torch.manual_seed(V)
    ld = (V + 7) // 8 * 8
    logits = (torch.randn(7, ld, device="cuda") * 3).bfloat16()[:, :V]
    labels = torch.full((7,), V - 1, device="cuda")
    logits[0, ::3] = float("-inf")
    logits[1, :V - 1] = float("-inf")
    logits[2, : V // 2] = -3.3895e38   # the type's lowest value
    logits[3, V // 2] = float("inf")
    logits[4, V // 3] = float("nan")
    logits[5] = float("-inf")
    labels[0], labels[6] = 1, 0
    loss, lse = _rows_fwd(logits, labels, -100)
    ref = torch.logsumexp(logits.double(), -1)
    want = ref - logits.double().gather(1, labels[:, None])[:, 0]
    for r in (0, 1, 2, 6):
        assert abs(lse[r].item() - ref[r].item()) <= 2e-6 * max(1.0, abs(ref[r].item()))
        assert abs(loss[r].item() - want[r].item()) <= 1e-5 * max(1.0, abs(want[r].item()))
    assert lse[3:6].isnan().all()


# fewer rows than a warp, more than a block, none that counts
@pytest.mark.parametrize("rows", [1, 31, 1025, 5000])
def test_cross_entropy_mean(rows):
    from nanopysche_b200.ops.xent import cross_entropy

    torch.manual_seed(rows)
    logits = torch.randn(rows, 16, device="cuda").bfloat16()
    labels = torch.randint(0, 16, (rows,), device="cuda")
    labels[::3] = -100
    ref = torch.nn.functional.cross_entropy(logits.double(), labels, ignore_index=-100, reduction="sum") / max(
        1, (labels != -100).sum().item())
    assert abs(cross_entropy(logits, labels).item() - ref.item()) <= 2e-6 * abs(ref.item())   # rows in fp32, few ulp each
    assert cross_entropy(logits, torch.full_like(labels, -100)).item() == 0


# one token, an odd number per CTA, more (head, slice) pairs than a block has threads, partial rotation
@pytest.mark.parametrize("B,S,hq,hkv,hd,rot", [(1, 1, 2, 1, 64, 64), (2, 333, 16, 8, 128, 128), (1, 77, 12, 12, 64, 32),
                                               (1, 40, 64, 64, 128, 128), (3, 1000, 4, 4, 64, 64)])
def test_qkv_rope_shapes(B, S, hq, hkv, hd, rot):
    from nanopysche_b200.ops.rope import apply_rope_ref, qkv_rope, rope_tables

    torch.manual_seed(S)
    qkv = torch.randn(B, S, (hq + 2 * hkv) * hd, device="cuda").bfloat16().requires_grad_(True)
    cos, sin = rope_tables(S + 5, rot, device="cuda")
    q, k, v = qkv_rope(qkv, cos, sin, hq, hkv, hd, pos_offset=5)
    x = qkv.detach().double().requires_grad_(True)
    h = x.view(B, S, hq + 2 * hkv, hd)
    c, s = cos.double()[5:5 + S][None, :, None], sin.double()[5:5 + S][None, :, None]
    a, b, rest = h[..., :rot // 2], h[..., rot // 2:rot], h[..., rot:]
    r = torch.cat([a * c - b * s, b * c + a * s, rest], -1)
    for got, want in ((q, r[:, :, :hq]), (k, r[:, :, hq:hq + hkv]), (v, h[:, :, hq + hkv:])):
        assert rel(got, want) < 4e-3
    gq, gk, gv = (torch.randn_like(t) for t in (q, k, v))
    torch.autograd.backward([q, k, v], [gq, gk, gv])
    torch.autograd.backward([r[:, :, :hq], r[:, :, hq:hq + hkv], h[:, :, hq + hkv:]], [gq.double(), gk.double(), gv.double()])
    assert rel(qkv.grad, x.grad) < 4e-3
    one = torch.cat([qkv.detach()[..., :hq * hd].unflatten(-1, (hq, hd))[:, :, :1]] * 2, 2)     # the framework's reference too
    ref = apply_rope_ref(one, cos, sin, 5)
    assert rel(ref[:, :, 0], q[:, :, 0]) < 4e-3 and torch.equal(ref[:, :, 0], ref[:, :, 1])


# both sides of the switches between the forms (2368 and 8192 tokens), T off whole groups of tokens, experts off a block of
# eight, D off a warp's 256 and off two of them
@pytest.mark.parametrize("T,D,E,K", [(5, 64, 4, 2), (2367, 256, 8, 2), (2371, 768, 8, 2), (4099, 2048, 12, 3), (2368, 1032, 8, 2),
                                     (8191, 264, 8, 2), (8193, 776, 9, 2)])
def test_router_forward_in_one_piece(T, D, E, K):
    from nanopysche_b200.models.moe import MoERouter, MoERouterConfig
    from nanopysche_b200.ops.moe import route

    torch.manual_seed(T)
    router = MoERouter(d_model=D, config=MoERouterConfig(num_experts=E, top_k=K, z_loss_multiplier=1e-2), device="cuda")
    x = torch.randn(T, D, device="cuda").bfloat16()
    w, idx, aux, counts = route(x, router)
    logits = x.double() @ router.gate.weight.double().t() + router.gate.bias.double()
    top, i64 = logits.topk(K, -1)
    assert (idx == i64).all(-1).float().mean() > 0.999           # a last-bit tie may go the other way
    same = (idx == i64).all(-1)
    assert rel(w[same], top.softmax(-1)[same]) < 1e-5
    f = torch.bincount(idx.reshape(-1), minlength=E).double() / T
    assert torch.equal(counts.long(), torch.bincount(idx.reshape(-1), minlength=E))
    ref = E * (f * logits.softmax(-1).mean(0)).sum() + 1e-2 * logits.logsumexp(-1).square().mean()
    assert abs(aux.item() - ref.item()) < 1e-5 * abs(ref.item())


def test_router_without_tokens():
    """No tokens: no error, counts and gradients of zero, and NaN as the mean over nothing."""
    from nanopysche_b200.ops.moe import _Router

    gate = [t.requires_grad_(True) for t in (torch.randn(4, 64, device="cuda"), torch.randn(4, device="cuda"))]
    x = torch.zeros(0, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w, idx, aux, counts = _Router.apply(x, *gate, None, 2, 0, 1e-2)
    assert w.shape == idx.shape == (0, 2) and aux.isnan() and counts.tolist() == [0] * 4
    w.sum().backward()
    assert x.grad.shape == (0, 64) and not gate[0].grad.any() and not gate[1].grad.any()


def test_auxiliary_losses_add_up_in_place():
    """``aux_loss`` is the caller's own tensor: scaling it and adding to it in place leave the gradients right."""
    from nanopysche_b200.models.moe import MoEBase

    torch.manual_seed(0)
    a, b = (MoEBase(d_model=128, hidden_size=256, num_experts=4, top_k=2, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    x = torch.randn(1, 200, 128, device="cuda").bfloat16()

    def grads(total):
        a.zero_grad(), b.zero_grad()
        total.backward()
        return [m.router.gate.weight.grad.clone() for m in (a, b)]

    (a(x), b(x))
    want = grads(2 * a.aux_loss + b.aux_loss)
    (a(x), b(x))
    total = a.aux_loss
    total.mul_(2)
    total += b.aux_loss
    for g, w in zip(grads(total), want):
        assert w.norm() > 0 and rel(g, w) < 1e-6


@pytest.mark.parametrize("fp8", [False, True])
def test_every_dispatch_starts_the_push_counters_anew(fp8):
    """Two rounds of dispatch and push (other tokens, other routing) give what a fresh runtime gives for the second one, the
    counters hold exactly that round's tiles, and a second push behind one dispatch is refused."""
    from nanopysche_b200.models.moe import MoEBase
    from nanopysche_b200.ops import _lib
    from nanopysche_b200.ops.moe import FusedMoERuntime

    T, D, H, E, K = 700, 256, 256, 8, 2
    torch.manual_seed(0)
    m = MoEBase(d_model=D, hidden_size=H, num_experts=E, top_k=K, dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        for w in (m.w1, m.w2, m.w3):
            w.normal_(0, 0.05)
        m.router.gate.weight.normal_()
    xs = [torch.randn(1, T, D, device="cuda").bfloat16() for _ in range(2)]

    def once(rt, x):
        m._fused_runtime = rt
        x = x.clone().requires_grad_(True)
        for p in m.parameters():
            p.grad = None
        rt.layer_index(m)
        y = m(x)
        fwd = rt.done_counters.clone()
        y.float().square().sum().backward()
        return [y.detach(), x.grad, m.w1.grad, m.w2.grad, m.w3.grad, fwd, rt.done_counters.clone(), rt.src_blocks.clone()]

    def runtime():
        return FusedMoERuntime(tokens=T, d_model=D, hidden=H, num_experts=E, top_k=K, n_layers=1, capacity_factor=None, fp8=fp8)

    rt = runtime()
    once(rt, xs[0])
    got, want = once(rt, xs[1]), once(runtime(), xs[1])
    for g, w in zip(got, want):
        assert torch.equal(g, w)
    assert got[-1].item() > 0 and got[5].item() % got[-1].item() == 0 and got[6].item() % got[-1].item() == 0
    with pytest.raises(_lib.KernelError, match="once behind every dispatch"):
        rt.grouped_gemm(rt.recv_g, m.w1, N=D, K=H, b_mn=True, group_stride_b=H, push_ptrs=rt.p_ret_g, push_epoch=1)
    _lib.check_status("after test")


def _plan(idx, E, cap):
    """The capacity rule on the host: a slot's position is its rank among the kept slots of its expert in token order; a token
    that any of its experts has no room for is dropped as a whole."""
    T, K = idx.shape
    hit = torch.zeros(T, E, dtype=torch.bool).scatter_(1, idx.long(), True)
    over = hit & (hit.cumsum(0) > cap) if cap >= 0 else torch.zeros_like(hit)
    keep = ~over.any(1)
    kept = hit & keep[:, None]
    pos = (kept.cumsum(0) - 1).gather(1, idx.long())
    pos[~keep] = -1
    return pos, keep, kept.sum(0), over.sum(0), (~keep).sum()


# the counters of the scan, in shared memory and (above 200 KB of indices) in memory, 16 and 32 bits wide
@pytest.mark.parametrize("T,cap,ranks", [(1, -1, 1), (1, 0, 1), (700, 150, 2), (4096, 1280, 4), (4096, -1, 8), (30000, 7000, 1),
                                         (70000, -1, 2), (70000, 20000, 4)])
def test_capacity_plan(T, cap, ranks):
    from nanopysche_b200.ops import _lib

    E, K = 8, 2
    torch.manual_seed(T)
    idx = torch.rand(T, E, device="cuda").topk(K, -1).indices.to(torch.int32)
    got = [torch.full(s, -7, device="cuda", dtype=torch.int32) for s in ((T, K), (T,), (E,), (E,), (1,))]
    sent = torch.empty(ranks, device="cuda", dtype=torch.int32)
    stats = torch.tensor([9, 100, 1000], device="cuda")
    _lib.call("capacity_plan", idx, T, E, K, cap, *got, sent, ranks, stats)
    want = _plan(idx.cpu(), E, cap)
    for g, w in zip(got, want):
        assert torch.equal(g.cpu().long().reshape(w.shape), w.long())
    assert torch.equal(sent.cpu().long(), want[2].view(ranks, -1).sum(1))
    d = want[4].item()
    assert stats.tolist() == [d, 100 + d, 1000 + T]


# single elements, vectors and tiles with remainders, more tiles than CTAs
@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1028, 8191, 8192 * 592 + 8197])
@pytest.mark.parametrize("copy16", [True, False])
def test_adamw_and_square_sum(n, copy16):
    from nanopysche_b200.ops import _lib

    torch.manual_seed(n)
    p, g, m = (torch.randn(n, device="cuda") for _ in range(3))
    v, w16 = torch.rand(n, device="cuda"), torch.zeros(n, device="cuda", dtype=torch.bfloat16)
    part = torch.full((_lib.lib().np_sumsq_parts(),), float("nan"), device="cuda")
    coef, lr, b1, b2, eps, wd, step = torch.tensor([0.5], device="cuda"), 1e-2, 0.9, 0.95, 1e-8, 0.1, 3
    P, G, M, V = p.double(), g.double() * 0.5, m.double(), v.double()
    _lib.call("sumsq", g, _lib.LL(n), part)
    _lib.call("adamw", p, g, m, v, w16 if copy16 else None, _lib.LL(n), lr, b1, b2, eps, wd, step, coef, None)
    # every square rounded once, then at most 32 additions per tile of a CTA and 13 over threads
    torch.testing.assert_close(part.double().sum(), g.double().square().sum(), rtol=(32 * (n // (8192 * 592) + 2) + 16) * 2 ** -24, atol=0)
    M, V = b1 * M + (1 - b1) * G, b2 * V + (1 - b2) * G * G
    P = P * (1 - lr * wd) - lr * (M / (1 - b1 ** step)) / ((V / (1 - b2 ** step)).sqrt() + eps)
    tol = dict(rtol=2 ** -20, atol=2 ** -20)      # some ten fp32 roundings of numbers of the size of one; 1 - b2^3 to 2^-21
    for got, want in ((p, P), (m, M), (v, V)):
        torch.testing.assert_close(got.double(), want, **tol)
    assert torch.equal(w16, p.bfloat16() if copy16 else torch.zeros_like(w16))


# one, two and more passes over the experts, picks per token that straddle the warps' runs, runs that stay in registers and longer ones
@pytest.mark.parametrize("T,E,K,cap", [(1, 1, 1, -1), (11, 2, 1, 3), (33, 31, 5, 4), (341, 32, 3, 40), (2731, 33, 3, 250),
                                       (1024, 64, 8, 128), (1025, 64, 8, 120), (1366, 65, 6, 100), (600, 130, 7, 30), (210000, 5, 1, 50000)])
def test_capacity_plan_of_many_experts(T, E, K, cap):
    from nanopysche_b200.ops import _lib

    torch.manual_seed(T)
    idx = torch.rand(T, E, device="cuda").topk(K, -1).indices.to(torch.int32)
    got = [torch.full(s, -7, device="cuda", dtype=torch.int32) for s in ((T, K), (T,), (E,), (E,), (1,))]
    _lib.call("capacity_plan", idx, T, E, K, cap, *got, None, 0, None)
    for g, w in zip(got, _plan(idx.cpu(), E, cap)):
        assert torch.equal(g.cpu().long().reshape(w.shape), w.long())


# widths that are no whole number of steps, more experts than a pass takes, both numbers of tokens per group at their edges
@pytest.mark.parametrize("T,D,E", [(1, 8, 1), (5, 264, 8), (9, 1032, 9), (1183, 768, 7), (1184, 768, 8), (1185, 768, 8), (1190, 2056, 17),
                                   (10000, 128, 64)])
def test_router_logits(T, D, E):
    from nanopysche_b200.ops import _lib

    torch.manual_seed(T)
    x, w = torch.randn(T, D, device="cuda").bfloat16(), torch.randn(E, D, device="cuda")
    bias, zero = torch.randn(E, device="cuda"), torch.ones(2 * E + 1, device="cuda", dtype=torch.int32)
    got = torch.full((T, E), float("nan"), device="cuda")
    _lib.call("router_logits", x, w, bias, got, T, D, E, zero, 2 * E)
    want = x.double() @ w.double().t() + bias.double()
    # fp32: each of the D products meets at most 8 additions a step, 5 + 2 over lanes and warps
    bound = (x.double().abs() @ w.double().abs().t() + bias.double().abs()) * (8 * -(-D // 1024) + 8) * 2 ** -24
    assert ((got.double() - want).abs() <= bound).all()
    assert zero[:-1].eq(0).all() and zero[-1] == 1
    # a token's sum does not depend on how many come with it
    few = torch.empty(min(T, 3), E, device="cuda")
    _lib.call("router_logits", x[-3:].contiguous(), w, bias, few, few.shape[0], D, E, None, 0)
    assert torch.equal(few, got[-3:])


# the order of a logit's sum: a lane's vectors one after the other, then the lanes in halves. One element per vector, so that the order
# within a vector does not count; magnitudes so far apart that any other order gives another result
@pytest.mark.parametrize("T,D,E", [(3, 2048, 8), (1184, 2048, 8), (1185, 2304, 5), (1200, 1024, 17)])
def test_router_logits_order_of_the_sum(T, D, E):
    from nanopysche_b200.ops import _lib

    torch.manual_seed(D)
    x, w = torch.zeros(T, D), torch.zeros(E, D)
    x[:, ::8] = torch.randn(T, D // 8) * 2.0 ** torch.randint(-6, 7, (T, D // 8))
    x = x.bfloat16()
    w[:, ::8] = torch.randn(E, D // 8) * 2.0 ** torch.randint(-6, 7, (E, D // 8))
    bias, got = torch.randn(E), torch.empty(T, E, device="cuda")
    _lib.call("router_logits", x.cuda(), w.cuda(), bias.cuda(), got, T, D, E, None, 0)
    t = x.float()[:, None, ::8] * w[None, :, ::8]                    # [T, E, vectors], one rounding each
    acc = torch.zeros(T, E, 32)
    for v in range(0, D // 8, 32):
        part = t[..., v:v + 32]
        acc[..., :part.shape[-1]] += part
    lane = torch.arange(32)
    for o in (16, 8, 4, 2, 1):
        acc = acc + acc[..., lane ^ o]
    assert torch.equal(got.cpu(), acc[..., 0] + bias)


# the ends of the exponent: sigmoid at subnormal numbers, at zero, one and infinity; each of the two reciprocal forms
def test_swiglu_at_the_ends_of_the_range():
    from nanopysche_b200.ops.activation import glu
    from nanopysche_b200.ops.gemm import gemm_glu_bwd, gemm_swiglu

    edge = torch.tensor([-3e38, -1e4, -100., -88.5, -88., -80., -20., -1., -0., 0., 1., 20., 88., 1e4, 3e38, -float("inf"),
                         float("inf"), float("nan")] + [0.5] * 6, device="cuda").bfloat16()
    F = edge.numel()
    gu = torch.cat([edge, torch.full_like(edge, 0.75)])[None].contiguous()
    h = glu(gu, "silu")
    g64 = edge.double()[None].requires_grad_(True)
    ref = torch.nn.functional.silu(g64) * 0.75
    # one rounding to bf16; the fp32 exponential overflows from 88.7 on, where silu is below 1e-36
    torch.testing.assert_close(h.double(), ref.detach(), rtol=2 ** -8, atol=1e-36, equal_nan=True)
    finite = edge.isfinite()
    x = gu.clone().requires_grad_(True)
    glu(x, "silu").backward(torch.ones_like(h))
    ref.sum().backward()
    torch.testing.assert_close(x.grad[0, :F][finite].double(), g64.grad[0][finite], rtol=2 ** -7, atol=1e-34)
    # the same pre-activations through the GEMM epilogues (identity weights keep them exactly)
    M = 256
    X = torch.zeros(M, F, device="cuda").bfloat16()
    X[:, :] = torch.where(finite, edge, torch.zeros_like(edge))
    eye = torch.eye(F, device="cuda").bfloat16()
    hh, pre = gemm_swiglu(X, eye, eye)
    x64 = X.double()
    keep = x64.abs() < 1e18   # the square of the rest leaves the range
    torch.testing.assert_close(hh.double()[keep], (torch.nn.functional.silu(x64) * x64)[keep], rtol=2 ** -7, atol=1e-34)
    one = torch.ones(M, F, device="cuda").bfloat16()
    d = gemm_glu_bwd(one, eye, torch.cat([X, 0.75 * one], 1).contiguous())
    want = torch.where(finite, g64.grad[0], torch.full_like(g64.grad[0], 0.375))
    torch.testing.assert_close(d[:, :F].double(), want.expand(M, F), rtol=2 ** -7, atol=1e-34)


# fewer heads than a warp holds, each of the three block sizes, one token, an odd number of tokens, more tokens than CTAs take twice
@pytest.mark.parametrize("B,S,hq,hkv", [(1, 1, 2, 1), (1, 77, 3, 3), (3, 777, 16, 8), (1, 1201, 32, 8), (2, 35, 40, 8), (1, 6, 56, 8)])
def test_qkv_norm_rope_backward(B, S, hq, hkv):
    from nanopysche_b200.ops.rope import qkv_norm_rope, rope_tables

    torch.manual_seed(S)
    qkv = torch.randn(B, S, (hq + 2 * hkv) * 128, device="cuda").bfloat16().requires_grad_(True)
    norms = [torch.nn.LayerNorm(128, device="cuda") for _ in range(2)]
    for m in norms:
        torch.nn.init.normal_(m.weight, 1.0, 0.2), torch.nn.init.normal_(m.bias, 0.0, 0.2)
    par = [p for m in norms for p in m.parameters()]
    cos, sin = rope_tables(S + 3, 128, device="cuda")
    out = qkv_norm_rope(qkv, *norms, cos, sin, hq, hkv, 3)
    g = [torch.randn_like(t) for t in out]
    got = torch.autograd.grad(out, [qkv, *par], g)
    x = qkv.detach().double().requires_grad_(True)
    p64 = [p.detach().double().requires_grad_(True) for p in par]
    h = x.view(B, S, hq + 2 * hkv, 128)
    n = [torch.nn.functional.layer_norm(t, (128,), *p64[2 * i:2 * i + 2], norms[i].eps) for i, t in enumerate((h[:, :, :hq], h[:, :, hq:hq + hkv]))]
    c, s = cos.double()[3:3 + S][None, :, None], sin.double()[3:3 + S][None, :, None]
    rot = [torch.cat([t[..., :64] * c - t[..., 64:] * s, t[..., 64:] * c + t[..., :64] * s], -1) for t in n]
    want = torch.autograd.grad([*rot, h[:, :, hq + hkv:]], [x, *p64], [t.double() for t in g])
    assert rel(got[0], want[0]) < 4e-3
    for a, b in zip(got[1:], want[1:]):      # fp32 sums over tokens and heads of bf16 terms
        assert rel(a, b) < 1e-4


# rows off a scale chunk of 128, one row, several column blocks; a row of zeros and the smallest and largest magnitudes
@pytest.mark.parametrize("rows,K", [(1, 128), (100, 384), (129, 256), (1000, 2816)])
def test_mx_quantiser_in_one_pass_with_swiglu(rows, K):
    from nanopysche_b200.ops.activation import glu
    from nanopysche_b200.ops.gemm_mxfp8 import mx_quantize, mx_quantize_glu, mx_quantize_ref

    torch.manual_seed(K)
    gu = (torch.randn(rows, 2 * K, device="cuda") * torch.exp2(torch.randint(-40, 20, (rows, 1), device="cuda").float())).bfloat16()
    gu[0, :K // 2] = 0
    x = gu[:, K:]
    for got, want in ((mx_quantize(x.contiguous()), mx_quantize_ref(x)), (mx_quantize(x), mx_quantize_ref(x))):
        assert torch.equal(got[0].view(torch.uint8), want[0].view(torch.uint8)) and torch.equal(got[1], want[1])
    q, sf, h = mx_quantize_glu(gu)
    two = mx_quantize(glu(gu))
    assert torch.equal(h, glu(gu)) and torch.equal(q.view(torch.uint8), two[0].view(torch.uint8)) and torch.equal(sf, two[1])


@pytest.mark.parametrize("rows,D,F", [(3, 128, 128), (200, 256, 384), (1030, 512, 1408)])
def test_mx_feed_forward_in_one_node(rows, D, F):
    """The same forward as the separate layers, bit for bit; gradients without the rounding of dh between them."""
    from nanopysche_b200.ops.activation import glu
    from nanopysche_b200.ops.gemm import feed_forward_glu, linear

    torch.manual_seed(F)
    x = torch.randn(rows, D, device="cuda").bfloat16().requires_grad_(True)
    w13, w2 = ((torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16().requires_grad_(True) for n, k in ((2 * F, D), (D, F)))
    w13._fp8_recipe = w2._fp8_recipe = "mxfp8"
    dy = torch.randn(rows, D, device="cuda").bfloat16()
    y, z = feed_forward_glu(x, w13, w2), linear(glu(linear(x, w13)), w2)
    assert type(y.grad_fn).__name__ == "_MXFeedForwardBackward" and torch.equal(y, z)
    for a, b in zip(torch.autograd.grad(y, [x, w13, w2], dy), torch.autograd.grad(z, [x, w13, w2], dy)):
        assert rel(a, b) < 6e-3      # bf16 roundings of dh, d gate and d up
    with torch.no_grad():
        assert torch.equal(feed_forward_glu(x, w13, w2), z)


# a chosen expert's part of the logit gradient is added to that of the auxiliary loss in one rounding
@pytest.mark.parametrize("T,E,K", [(33, 3, 1), (300, 8, 2), (200, 17, 4), (130, 64, 8)])
def test_router_logit_gradient_is_added_in_one_rounding(T, E, K):
    from nanopysche_b200.ops import _lib

    torch.manual_seed(E)
    logits, f, daux = torch.randn(T, E, device="cuda"), torch.rand(E, device="cuda"), torch.randn(1, device="cuda") * T
    top, idx = logits.topk(K, -1)
    w, dw, idx = top.softmax(-1).contiguous(), torch.randn(T, K, device="cuda") * 0.1, idx.to(torch.int32)
    dl = torch.empty(2, T, E, device="cuda")
    for out, d in zip(dl, (None, dw)):
        _lib.call("router_bwd", logits, None, w, idx, d, f, daux, 1.0, 0.01, out, T, E, K, 0)
    aux, got, w, dw = (t.cpu().double() for t in (*dl, w, dw))
    fma = lambda a, b, c: (a * b + c).float().double()      # the product of two floats is exact in 64 bits  # noqa: E731
    wsum = torch.zeros(T, dtype=torch.double)
    for k in range(K):
        wsum = fma(w[:, k], dw[:, k], wsum)
    want = aux.clone()
    for k in range(K):
        at = (torch.arange(T), idx[:, k].cpu().long())
        want[at] = fma(w[:, k], (dw[:, k] - wsum).float().double(), want[at])
    assert torch.equal(got, want)


# the means of a head in the backward of head norms: eight neighbouring columns one after the other, then those groups in halves. Zero
# inputs leave the first mean alone; pairs of +-2^24 beside small whole numbers make every other order another whole number
@pytest.mark.parametrize("T,hq,hkv", [(3, 2, 1), (300, 16, 8), (200, 32, 8), (90, 40, 16)])
def test_head_norm_backward_order_of_the_means(T, hq, hkv):
    from nanopysche_b200.ops import rope as R

    torch.manual_seed(T)
    H = hq + hkv
    d = torch.zeros(T, H, 128)
    at = torch.rand(T, H, 128).topk(16, -1).indices
    d.scatter_(2, at, torch.cat([torch.randint(1, 9, (T, H, 10)).float(), torch.tensor([1., -1., 1., -1., 1., -1.]).expand(T, H, 6) * 2 ** 24], -1))
    qkv = torch.zeros(1, T, (H + hkv) * 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    norms = [torch.nn.LayerNorm(128, eps=2.0 ** -16, device="cuda") for _ in range(2)]
    cos, sin = R.rope_tables(4, 128, device="cuda")
    ids = torch.zeros(1, T, device="cuda", dtype=torch.int32)      # position 0: no rotation
    q, k, _ = R.qkv_norm_rope(qkv, *norms, cos, sin, hq, hkv, 0, ids)
    g = d.cuda().bfloat16()[None]
    torch.autograd.backward([q, k], [g[:, :, :hq].contiguous(), g[:, :, hq:].contiguous()])
    t = (d[..., :64] + d[..., 64:]).view(T, H, 8, 8)
    acc = torch.zeros(T, H, 8)
    for j in range(8):
        acc = acc + t[..., j]
    i = torch.arange(8)
    for o in (1, 2, 4):
        acc = acc + acc[..., i ^ o]
    want = 256.0 * (d - acc[..., :1] / 128)
    got = qkv.grad[0, :, :H * 128].view(T, H, 128).float().cpu()
    assert ((got - want).abs() <= want.abs() * 2.0 ** -7).all()


# the order of the gradient norm's sums: a thread's vectors one after the other, lanes in halves, warps in halves. One element per
# vector, so that the order within a vector does not count
@pytest.mark.parametrize("n", [3, 40, 151552 * 4, 151552 * 4 * 9 + 4003])
def test_sum_of_squares_order(n):
    from nanopysche_b200.ops import _lib

    torch.manual_seed(n)
    parts = _lib.lib().np_sumsq_parts()
    x = torch.zeros(n)
    x[::4] = torch.randn(-(-n // 4)) * 2.0 ** torch.randint(-6, 7, (-(-n // 4),))
    tail = x[n // 4 * 4:]
    got = torch.zeros(parts, device="cuda")
    _lib.call("sumsq", x.cuda(), _lib.LL(n), got)
    t = (x * x)[:n // 4 * 4:4]
    s = torch.zeros(parts * 256)
    for k in range(0, t.numel(), parts * 256):
        s[:t[k:k + parts * 256].numel()] += t[k:k + parts * 256]
    s[0] += (tail * tail).sum()                      # at most one of them is not zero
    s, i = s.view(parts, 8, 32), torch.arange(32)
    for o in (16, 8, 4, 2, 1):
        s = s + s[..., i ^ o]
    s = torch.nn.functional.pad(s[..., 0], (0, 24))
    for o in (16, 8, 4, 2, 1):
        s = s + s[..., i ^ o]
    assert torch.equal(got.cpu(), s[:, 0])


# the order of the gate's gradient: chunks of 64 tokens, of a chunk every fourth token by one lane, lanes 0 + 2 and 1 + 3, the chunks in eight
# sums; the bias gradient in 1024 / E groups of rows. Both sizes of CTA, one and more passes over the experts, a last chunk that is short
@pytest.mark.parametrize("T,D,E", [(1, 8, 1), (70, 136, 3), (600, 16, 8), (1025, 8, 17), (1500, 24, 5)])
def test_router_gate_gradient_order(T, D, E):
    from nanopysche_b200.ops import _lib

    torch.manual_seed(T)
    dl, x = torch.randn(T, E) * 2.0 ** torch.randint(-4, 5, (T, 1)), torch.randn(T, D).bfloat16()
    w, b = torch.full((2, E, D), 0.5, device="cuda"), torch.full((2, E), 0.5, device="cuda")
    scratch = torch.empty((T + 63) // 64 * E * D + 1024, device="cuda")
    for acc in (0, 1):
        _lib.call("router_dgate", dl.cuda(), x.cuda(), w[acc], b[acc], scratch, T, D, E, acc)
    chunks = (T + 63) // 64
    pad = lambda t: torch.nn.functional.pad(t, (0, 0, 0, chunks * 64 - T)).view(chunks, 16, 4, -1)      # noqa: E731
    l, v = pad(dl).double(), pad(x.float()).double()
    part = torch.zeros(chunks, 4, E, D)
    for i in range(16):                 # one rounding for each product and its addition
        part = (part.double() + l[:, i, :, :, None] * v[:, i, :, None, :]).float()
    part = (part[:, 0] + part[:, 2]) + (part[:, 1] + part[:, 3])
    a = torch.zeros(8, E, D)
    whole = chunks // 8 * 8
    for p in range(chunks):
        a[p % 8 if p < whole else 0] += part[p]
    want = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]))
    groups = 1024 // E
    a4 = torch.zeros(groups, 4, E)
    for r in range(T):
        g, i = r % groups, r // groups
        rows = (T - g + groups - 1) // groups          # of this group
        a4[g, i % 4 if i < rows // 4 * 4 else 0] += dl[r]
    s = (a4[:, 0] + a4[:, 1]) + (a4[:, 2] + a4[:, 3])
    bias = torch.zeros(E)
    for g in range(groups):
        bias = bias + s[g]
    assert torch.equal(w.cpu(), torch.stack([want, want + 0.5])) and torch.equal(b.cpu(), torch.stack([bias, bias + 0.5]))


# the Python form of the expert layer, which runs with peers, and the native one: the same kernels and bits on one rank. Capacity with drops,
# gradients into main_grad and into tensors, a shared expert's output
@pytest.mark.parametrize("T,E,K,capacity,arena,shared", [(520, 8, 2, None, True, 0), (1030, 4, 2, 1.25, True, 1), (300, 8, 1, 1.5, False, 0)])
def test_expert_layer_forms_agree(T, E, K, capacity, arena, shared, monkeypatch):
    from nanopysche_b200.engine import prepare_training
    from nanopysche_b200.models.moe import MoEBase
    from nanopysche_b200.ops import moe as ops

    D, H = 256, 512
    out = []
    for native in (True, False):
        monkeypatch.setattr(ops, "_native_form", lambda rt: native)
        torch.manual_seed(T)
        m = MoEBase(d_model=D, hidden_size=H, num_experts=E, top_k=K, capacity_factor=capacity, shared_expert=bool(shared),
                    dtype=torch.bfloat16, device="cuda")
        with torch.no_grad():
            for w in m.parameters():
                w.normal_(0, 0.05)
        if arena:
            _, a = prepare_training(m, tokens_per_rank=T, lr=1e-3)
        else:
            ops.build_runtime([m], tokens=T, device=torch.device("cuda"))
        x = torch.randn(1, T, D, device="cuda").bfloat16().requires_grad_(True)
        dy = torch.randn(1, T, D, device="cuda").bfloat16()
        for _ in range(2):
            x.grad = None
            y = m(x)
            y.backward(dy)
        grads = dict(a.named_main_grads()) if arena else {n: p.grad for n, p in m.named_parameters()}
        out.append([y, x.grad, m._per_expert_drop_counts, *(g for g in grads.values() if g is not None)])
    assert len(out[0]) == len(out[1]) > 5 and all(torch.equal(p, q) for p, q in zip(*out))


def test_native_expert_layer_asks_before_it_pushes():
    """Every pushing product of the native layer takes its counters from the runtime, which refuses a second one behind a dispatch."""
    from nanopysche_b200.models.moe import MoEBase
    from nanopysche_b200.ops import _lib
    from nanopysche_b200.ops.moe import build_runtime

    m = MoEBase(d_model=256, hidden_size=256, num_experts=4, top_k=2, dtype=torch.bfloat16, device="cuda")
    rt = build_runtime([m], tokens=300, device=torch.device("cuda"))
    asked, ask = [], rt._push_counters
    rt._push_counters = lambda: (asked.append(rt._may_push), ask())[1]
    x = torch.randn(1, 300, 256, device="cuda").bfloat16().requires_grad_(True)
    m(x).sum().backward()
    assert asked == [True, True] and not rt._may_push                 # forward and backward, each behind a dispatch of its own
    with pytest.raises(_lib.KernelError, match="once behind every dispatch"):
        rt._push_counters()
