"""The two-CTA GEMM kernel (256 x 256 tiles, K whole or in parts) in every layout and epilogue it takes, against fp32
PyTorch products (GPU only). fp32 outputs of bf16 operands: the products are exact in fp32, the sums of K of them carry
about sqrt(K) 2^-24 relative to the terms; 2e-5 is an order above that at the largest K here. bf16 outputs: 3e-3."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b.double()).norm() / (b.double().norm() + 1e-30)).item()


@pytest.fixture(autouse=True)
def _status_clean():
    from nanopysche_b200.ops import _lib

    yield
    torch.cuda.synchronize()
    _lib.check_status("after test")


# edges of the 256-row tiles, of the 64-wide K steps and of the staged output boxes (32 rows, 32 / 64 columns)
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (264, 264, 520), (520, 136, 1000), (129, 40, 4096), (776, 2312, 512)])
@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("layout", ["fwd", "dgrad", "wgrad"])
def test_pair_gemm(M, N, K, split, layout):
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(M + N + K)
    a_mn, b_mn = layout == "wgrad", layout != "fwd"
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    ref = a.float() @ b.float().t()
    if a_mn and M % 8:
        a = torch.nn.functional.pad(a, (0, 0, 0, -M % 8))
        ref = a.float() @ b.float().t()
    A, B = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    kw = dict(a_mn=a_mn, b_mn=b_mn, bn=256, mt=2, split=split)
    assert rel(gemm(A, B, **kw), ref) < 3e-3
    y = gemm(A, B, out_dtype=torch.float32, **kw)
    assert rel(y, ref) < 2e-5
    assert torch.equal(y, gemm(A, B, out_dtype=torch.float32, **kw))          # the same bits every time
    acc = torch.randn_like(y)
    want = acc.double() + 0.5 * ref.double()
    gemm(A, B, out=acc, accumulate=True, alpha=0.5, **kw)
    assert rel(acc, want) < 2e-5
    bias = torch.randn(N, device="cuda")
    assert rel(gemm(A, B, bias=bias, out_dtype=torch.float32, **kw), ref + bias) < 2e-5


# tiles of 128 and 192 columns: half of 192 is one and a half of the 64-column chunks that an MN-major B is loaded in
@pytest.mark.parametrize("M,N,K", [(256, 192, 64), (264, 264, 520), (520, 136, 1000), (129, 40, 4096), (776, 2312, 512)])
@pytest.mark.parametrize("layout", ["fwd", "dgrad", "wgrad"])
@pytest.mark.parametrize("pair_bn", [128, 192])
def test_pair_gemm_narrow_tiles(M, N, K, layout, pair_bn):
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(M + N + K)
    a_mn, b_mn = layout == "wgrad", layout != "fwd"
    M += -M % 8 if a_mn else 0
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    ref = a.float() @ b.float().t()
    A, B = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    kw = dict(a_mn=a_mn, b_mn=b_mn, pair_bn=pair_bn)
    assert rel(gemm(A, B, **kw), ref) < 3e-3
    acc = torch.randn(M, N, device="cuda")
    want = acc.double() + 0.5 * ref.double()
    gemm(A, B, out=acc, accumulate=True, alpha=0.5, **kw)
    assert rel(acc, want) < 2e-5
    wide = torch.full((M, N + 24), 7.0, device="cuda").bfloat16()      # rows of a wider buffer: nothing beside them is written
    gemm(A, B, out=wide[:, :N], **kw)
    assert rel(wide[:, :N], ref) < 3e-3 and (wide[:, N:] == 7).all()
    y = gemm(A, B, out_dtype=torch.float32, **kw)
    assert rel(y, ref) < 2e-5 and torch.equal(y, gemm(A, B, out_dtype=torch.float32, **kw))


@pytest.mark.parametrize("M,F,K", [(256, 192, 64), (300, 264, 200), (1000, 704, 512)])
@pytest.mark.parametrize("pair_bn", [128, 192, 256])
def test_pair_glu_bwd_tiles(M, F, K, pair_bn):
    from nanopysche_b200.ops.gemm import gemm_glu_bwd

    torch.manual_seed(F)
    dy, w2 = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(K, F, device="cuda") * K ** -0.5).bfloat16()
    gu = torch.randn(M, 2 * F, device="cuda").bfloat16()
    g, u = (t.float().requires_grad_(True) for t in gu.chunk(2, 1))
    (torch.nn.functional.silu(g) * u).backward(dy.float() @ w2.float())
    assert rel(gemm_glu_bwd(dy, w2, gu, pair_bn=pair_bn), torch.cat([g.grad, u.grad], 1)) < 3e-3


# both gradients of a linear layer in one launch: either contraction the longer one, fewer tiles than pairs of CTAs and several
# rounds of them that do not come out even, M at which a choice of its own is made, sizes off the tiles
@pytest.mark.parametrize("T,N,K", [(264, 136, 200), (136, 1032, 264), (2048, 1024, 1024), (2331, 2048, 2048), (4096, 2304, 768), (300, 8200, 1000)])
@pytest.mark.parametrize("pair_bn", [0, 128, 192, 256])
def test_two_gradients_in_one_launch(T, N, K, pair_bn):
    from nanopysche_b200.ops.gemm import gemm_dgrad_wgrad, gemm_glu_bwd

    torch.manual_seed(T + N)
    dy, x = torch.randn(T, N, device="cuda").bfloat16(), torch.randn(T, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * N ** -0.5).bfloat16()
    acc = torch.randn(N, K, device="cuda")
    want = dy.float().t() @ x.float()
    for out, add in ((None, None), (torch.full_like(acc, float("nan")), None), (acc.clone(), acc)):
        dx, dw = gemm_dgrad_wgrad(dy, w, x, out=out, accumulate=add is not None, pair_bn=pair_bn)
        assert rel(dx, dy.float() @ w.float()) < 3e-3
        assert rel(dw, want if add is None else want + add) < (3e-3 if out is None else 2e-5)
        dx2, dw2 = gemm_dgrad_wgrad(dy, w, x, out=None if out is None else (torch.empty_like(acc) if add is None else add.clone()),
                                    accumulate=add is not None, mt=2)      # two launches
        assert rel(dx, dx2) < 2e-3 and rel(dw, dw2) < (2e-3 if out is None else 1e-6)
    gu = torch.randn(T, 2 * K, device="cuda").bfloat16()
    dgu, dw = gemm_dgrad_wgrad(dy, w, x, out=torch.empty_like(acc), gu=gu, pair_bn=pair_bn)
    assert rel(dgu, gemm_glu_bwd(dy, w, gu)) < 2e-3 and rel(dw, want) < 2e-5


@pytest.mark.parametrize("M,F,K", [(256, 128, 64), (300, 264, 200), (1000, 704, 512)])
def test_pair_swiglu(M, F, K):
    from nanopysche_b200.ops.gemm import gemm_swiglu

    torch.manual_seed(F)
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = torch.randn(2 * F, K, device="cuda").bfloat16() * K ** -0.5
    h, gu = gemm_swiglu(x, w[:F], w[F:])
    g, u = x.float() @ w[:F].float().t(), x.float() @ w[F:].float().t()
    assert rel(gu, torch.cat([g, u], 1)) < 3e-3 and rel(h, torch.nn.functional.silu(g) * u) < 3e-3


@pytest.mark.parametrize("M,N,K", [(4096, 768, 768), (768, 768, 4096), (2304, 768, 4096), (4096, 2304, 768), (200, 3000, 72)])
def test_chosen_kernel_agrees_with_the_one_cta_tile(M, N, K):
    """Whatever the cost rule picks: the fp32 result differs from the 128 x 128 tile's by the order of the sums only."""
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(N)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    assert rel(gemm(a, b, out_dtype=torch.float32), gemm(a, b, out_dtype=torch.float32, bn=128)) < 1e-6 * K ** 0.5


@pytest.mark.parametrize("M,F,D", [(256, 256, 64), (130, 264, 200), (1000, 712, 512), (4096, 768, 768)])
@pytest.mark.parametrize("kw", [dict(bn=0), dict(bn=256, mt=1), dict(bn=256, mt=2), dict(bn=128)])
def test_swiglu_backward_epilogue(M, F, D, kw):
    """``dh = dy @ w2`` taken to ``[d gate | d up]`` inside the GEMM; bf16 results of fp32 values: 3e-3."""
    import ctypes as C

    from nanopysche_b200.ops import _lib

    torch.manual_seed(F)
    dy = torch.randn(M, D, device="cuda").bfloat16()
    w2 = (torch.randn(D, F, device="cuda") * D ** -0.5).bfloat16()
    gu = torch.randn(M, 2 * F, device="cuda").bfloat16()
    out = torch.full((M, 2 * F), float("nan"), device="cuda", dtype=torch.bfloat16)
    a = _lib.GemmArgs()
    a.A, a.B, a.C, a.C2 = dy.data_ptr(), w2.data_ptr(), out.data_ptr(), gu.data_ptr()
    a.lda, a.ldb, a.ldc, a.ldc2, a.a_rows, a.b_rows = D, F, 2 * F, 2 * F, M, D
    a.M, a.N, a.K, a.b_mn, a.epilogue, a.alpha = M, F, D, 1, 2, 1.0
    a.bn, a.mt = kw["bn"], kw.get("mt", 0)
    assert _lib.lib().np_gemm_bf16(C.byref(a), C.c_void_p(_lib.stream())) == 0
    g64 = gu.double().requires_grad_(True)
    h = torch.nn.functional.silu(g64[:, :F]) * g64[:, F:]
    h.backward(dy.double() @ w2.double())
    assert rel(out, g64.grad) < 3e-3


@pytest.mark.parametrize("M,N,H", [(256, 256, 64), (300, 264, 192), (1000, 520, 704)])
@pytest.mark.parametrize("mt", [1, 2])
def test_contraction_over_two_weights_and_rows_into_two_outputs(M, N, H, mt):
    import ctypes as C

    from nanopysche_b200.ops import _lib

    torch.manual_seed(H)
    a2 = torch.randn(M, 2 * H, device="cuda").bfloat16()
    w1, w3 = (torch.randn(H, N, device="cuda").bfloat16() for _ in range(2))
    out = torch.empty(M, N, device="cuda")
    g = _lib.GemmArgs()
    g.A, g.B, g.B2, g.C = a2.data_ptr(), w1.data_ptr(), w3.data_ptr(), out.data_ptr()
    g.lda, g.ldb, g.ldc, g.a_rows, g.b_rows = 2 * H, N, N, M, H
    g.M, g.N, g.K, g.b_mn, g.out_f32, g.alpha, g.k_split, g.bn, g.mt = M, N, 2 * H, 1, 1, 1.0, H, 256, mt
    assert _lib.lib().np_gemm_bf16(C.byref(g), C.c_void_p(_lib.stream())) == 0
    assert rel(out, a2[:, :H].double() @ w1.double() + a2[:, H:].double() @ w3.double()) < 2e-5

    K, rows = M, 256                                # two outputs of 256 rows each from one transposed operand
    x = torch.randn(K, N, device="cuda").bfloat16()
    two = torch.randn(K, 2 * rows, device="cuda").bfloat16()
    for acc in (0, 1):
        o1, o2 = torch.ones(rows, N, device="cuda"), torch.ones(rows, N, device="cuda")
        g = _lib.GemmArgs()
        g.A, g.B, g.C, g.C2 = two.data_ptr(), x.data_ptr(), o1.data_ptr(), o2.data_ptr()
        g.lda, g.ldb, g.ldc, g.a_rows, g.b_rows = 2 * rows, N, N, K, K
        g.M, g.N, g.K, g.a_mn, g.b_mn, g.out_f32, g.alpha = 2 * rows, N, K, 1, 1, 1, 1.0
        g.accumulate, g.m_split, g.bn, g.mt = acc, rows, 256, mt
        assert _lib.lib().np_gemm_bf16(C.byref(g), C.c_void_p(_lib.stream())) == 0
        ref = two.double().t() @ x.double() + acc
        assert rel(o1, ref[:rows]) < 2e-5 and rel(o2, ref[rows:]) < 2e-5


def test_feed_forward_without_gradients_and_of_frozen_weights():
    from nanopysche_b200.ops.gemm import feed_forward_glu

    torch.manual_seed(2)
    x = torch.randn(2, 70, 128, device="cuda").bfloat16()
    w13, w2 = (torch.randn(512, 128, device="cuda") * 0.1).bfloat16(), (torch.randn(128, 256, device="cuda") * 0.1).bfloat16()
    with torch.no_grad():
        y = feed_forward_glu(x, w13, w2)
    xa = x.clone().requires_grad_(True)
    ya = feed_forward_glu(xa, w13, w2)
    ya.sum().backward()
    x64 = x.double().requires_grad_(True)
    gu = x64 @ w13.double().t()
    y64 = (torch.nn.functional.silu(gu[..., :256]) * gu[..., 256:]) @ w2.double().t()
    y64.sum().backward()
    assert torch.equal(y, ya) and rel(y, y64) < 6e-3 and rel(xa.grad, x64.grad) < 1e-2


# rows that do not start on 16-byte boundaries: odd widths on both sides of the few-row switch (64 rows) and of the 128-row tiles,
# an aligned width behind an odd base, a row stride below a vector's, aligned rows of a length that is no whole number of vectors
@pytest.mark.parametrize("M", [5, 65, 130, 700])
@pytest.mark.parametrize("N,off,ld", [(1003, 0, 1003), (129, 0, 129), (2052, 0, 2052), (512, 1, 520), (1001, 3, 1010), (7, 0, 7),
                                      (13, 0, 16), (207, 8, 208), (100, 0, 112), (1030, 0, 1048)])
@pytest.mark.parametrize("kw", [dict(), dict(bn=128), dict(bn=256, mt=1), dict(bn=256, mt=2), dict(bn=256, mt=2, split=2)])
def test_outputs_with_unaligned_rows(M, N, off, ld, kw):
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(M + N)
    K = 512
    x, w = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    ref = x.double() @ w.double().t()
    bias = torch.randn(N, device="cuda")
    for dt, tol in ((torch.bfloat16, 3e-3), (torch.float32, 2e-5)):
        def view(fill):
            buf = torch.full((M * ld + off + 8,), fill, device="cuda", dtype=dt)
            return buf, buf[off:off + M * ld].view(M, ld)[:, :N]

        buf, out = view(7.0)
        gemm(x, w, out=out, bias=bias, **kw)
        assert rel(out, ref + bias.double()) < tol
        rest = torch.ones_like(buf, dtype=torch.bool)                  # nothing beside the rows is written
        rest[off:off + M * ld].view(M, ld)[:, :N] = False
        assert (buf[rest] == 7.0).all()
        _, acc = view(1.5)
        gemm(x, w, out=acc, accumulate=True, **kw)
        assert rel(acc, ref + 1.5) < tol
        _, res = view(0.25)
        assert rel(gemm(x, w, residual=res, out_dtype=dt, **kw), ref + 0.25) < tol


@pytest.mark.parametrize("M,F", [(65, 100), (300, 1003), (700, 129), (256, 260)])
def test_swiglu_with_unaligned_rows(M, F):
    from nanopysche_b200.ops.gemm import gemm_swiglu

    torch.manual_seed(F)
    x, w = torch.randn(M, 128, device="cuda").bfloat16(), (torch.randn(2 * F, 128, device="cuda") * 0.1).bfloat16()
    h, gu = gemm_swiglu(x, w[:F], w[F:])
    g, u = x.double() @ w[:F].double().t(), x.double() @ w[F:].double().t()
    assert rel(gu, torch.cat([g, u], 1)) < 3e-3 and rel(h, torch.nn.functional.silu(g) * u) < 3e-3


def test_feed_forward_of_mismatched_widths_is_refused():
    from nanopysche_b200.ops.gemm import feed_forward_glu, gemm_swiglu

    x = torch.randn(2, 70, 128, device="cuda").bfloat16()
    w13, w2 = torch.randn(512, 64, device="cuda").bfloat16(), torch.randn(128, 256, device="cuda").bfloat16()
    with pytest.raises(AssertionError, match="contraction"):
        feed_forward_glu(x, w13, w2)
    with pytest.raises(AssertionError, match="contraction"):
        feed_forward_glu(x, torch.randn(256, 128, device="cuda").bfloat16(), w2)     # w2 of another hidden size
    with pytest.raises(AssertionError):
        gemm_swiglu(x[0], w13[:256].t(), w13[256:].t())


def _kernels(f):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    return " ".join(e.key for e in p.key_averages())


# a launch of one CTA has no pair; a request without a tile width still decides the kernel
@pytest.mark.parametrize("kw,pair", [(dict(bn=256, mt=2, max_ctas=1), False), (dict(bn=256, mt=2, max_ctas=3), True),
                                     (dict(mt=2), True), (dict(mt=1), False), (dict(split=2), True), (dict(split=4, mt=2), True),
                                     (dict(bn=256, split=2), True), (dict(bn=128, mt=2), False)])
def test_the_kernel_asked_for_runs(kw, pair):
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(1)
    a, b = torch.randn(300, 512, device="cuda").bfloat16(), torch.randn(520, 512, device="cuda").bfloat16()
    out = torch.full((300, 520), float("nan"), device="cuda")
    gemm(a, b, out=out, **kw)
    assert rel(out, a.double() @ b.double().t()) < 2e-5
    assert ("pair" in _kernels(lambda: gemm(a, b, out=out, **kw))) == pair


# the expert layer's backward with two products per launch: regions of several row blocks, uneven and empty experts, a capacity that
# drops tokens, gradients into new tensors and added to main_grad
@pytest.mark.parametrize("T,E,K,capacity", [(1000, 4, 2, None), (1536, 8, 2, 1.25), (2050, 16, 1, None), (520, 4, 4, 2.0)])
def test_expert_layer_backward_against_64_bits(T, E, K, capacity):
    from nanopysche_b200.engine import prepare_training
    from nanopysche_b200.models.moe import MoEBase

    D, H = 256, 512
    torch.manual_seed(T)
    m = MoEBase(d_model=D, hidden_size=H, num_experts=E, top_k=K, capacity_factor=capacity, dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        for w in (m.w1, m.w2, m.w3, m.router.gate.weight):
            w.normal_(0, 0.05)
        if K < E:
            m.router.gate.bias.zero_()[-1] = -30.0      # an expert without tokens
    _, arena = prepare_training(m, tokens_per_rank=T, lr=1e-3)
    x = torch.randn(1, T, D, device="cuda").bfloat16().requires_grad_(True)
    dy = torch.randn(1, T, D, device="cuda").bfloat16() * 0.1
    for _ in range(2):      # the second pass adds to the gradients of the first
        x.grad = None
        m(x).backward(dy)
    p = {n: w.detach().double().requires_grad_(True) for n, w in m.named_parameters()}
    x64 = x.detach().double()[0].requires_grad_(True)
    logits = x64 @ p["router.gate.weight"].t() + p["router.gate.bias"]
    top, idx = logits.topk(K, -1)
    gate, hit = top.softmax(-1), torch.zeros(T, E, device="cuda", dtype=torch.double).scatter_(1, idx, 1.0)
    keep = torch.ones(T, device="cuda", dtype=torch.bool) if capacity is None else ~((hit > 0) & (hit.cumsum(0) > int(capacity * T / E))).any(1)
    y = torch.zeros_like(x64)
    for e in range(E):
        t, k = ((idx == e) & keep[:, None]).nonzero(as_tuple=True)
        r = slice(e * H, (e + 1) * H)
        he = torch.nn.functional.silu(x64[t] @ p["w1"][r].t()) * (x64[t] @ p["w3"][r].t())
        y = y.index_add(0, t, he @ p["w2"][r] * gate[t, k][:, None])
    want = torch.autograd.grad(y, [x64, *(p[n] for n in ("w1", "w2", "w3"))], dy.double()[0])
    assert rel(x.grad[0], want[0]) < 1.5e-2          # bf16 activations and gradients between five products
    main = dict(arena.named_main_grads())
    for n, g in zip(("w1", "w2", "w3"), want[1:]):
        assert rel(main[n].view(g.shape), 2 * g) < 1.5e-2


# outputs whose sum over K is cut into 1, 2 and 4 parts (the cut is a rule of the sizes): every kernel that forms such a sum gives its
# bits, in one pair of CTAs or over a cluster, stored by TMA and from registers, alone and beside another product in a launch
@pytest.mark.parametrize("M,N,K", [(1024, 1024, 2048), (768, 768, 4096), (2048, 1024, 3072), (520, 136, 1000), (129, 40, 4096)])
@pytest.mark.parametrize("split", [2, 4])
@pytest.mark.parametrize("layout", ["fwd", "dgrad", "wgrad"])
def test_parts_of_a_sum_in_one_pair(M, N, K, split, layout):
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(M + N + K)
    a_mn, b_mn = layout == "wgrad", layout != "fwd"
    M += -M % 8 if a_mn else 0
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    ref = a.float() @ b.float().t()
    A, B = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    acc = torch.randn(M, N, device="cuda")
    for kw in (dict(), dict(out_dtype=torch.float32), dict(accumulate=True, alpha=0.5)):
        new = {"out": acc.clone()} if "accumulate" in kw else {}
        y = gemm(A, B, a_mn=a_mn, b_mn=b_mn, pair_bn=128, split=split, **kw, **new)
        new = {"out": acc.clone()} if "accumulate" in kw else {}
        z = gemm(A, B, a_mn=a_mn, b_mn=b_mn, split=split, **kw, **new)
        want = acc.double() + 0.5 * ref.double() if "accumulate" in kw else ref
        assert torch.equal(y, z) and rel(y, want) < (3e-3 if y.dtype == torch.bfloat16 else 2e-5)


@pytest.mark.parametrize("T,N,K", [(2048, 1024, 1024), (2048, 5632, 1024), (2048, 3072, 1024), (4096, 768, 768), (4096, 2304, 768),
                                   (2331, 2048, 4096), (640, 512, 2048), (136, 1032, 264)])
@pytest.mark.parametrize("pair_bn", [0, 128, 192, 256])
def test_gradients_do_not_depend_on_what_shares_their_launch(T, N, K, pair_bn):
    """A frozen weight or a deferred weight gradient leaves the bits of the input gradient as they are, and the other way round."""
    from nanopysche_b200.ops.gemm import gemm, gemm_dgrad_wgrad

    torch.manual_seed(T + N)
    dy, x = torch.randn(T, N, device="cuda").bfloat16(), torch.randn(T, K, device="cuda").bfloat16()
    w, acc = (torch.randn(N, K, device="cuda") * N ** -0.5).bfloat16(), torch.randn(N, K, device="cuda")
    dx, dw = gemm_dgrad_wgrad(dy, w, x, out=acc.clone(), accumulate=True, pair_bn=pair_bn)
    assert torch.equal(dx, gemm(dy, w, b_mn=True))
    assert torch.equal(dw, gemm(dy, x, a_mn=True, b_mn=True, out=acc.clone(), accumulate=True))


# Cuts of a sum over K, whatever kernel runs it: by the sizes alone. (M, N, K): parts
CUTS = {(768, 768, 4096): 4, (2304, 768, 4096): 2, (2048, 1024, 3072): 2, (1024, 1024, 2048): 2, (2048, 1024, 2816): 2, (200, 6144, 4096): 2,
        (4096, 768, 768): 1, (2048, 3072, 1024): 1, (3072, 1024, 2048): 1, (2331, 2048, 4096): 1}


@pytest.mark.parametrize("shape,parts", CUTS.items())
def test_where_a_sum_is_cut(shape, parts):
    from nanopysche_b200.ops.gemm import gemm

    M, N, K = shape
    torch.manual_seed(K)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    y = gemm(a, b, out_dtype=torch.float32)
    same = {p: torch.equal(y, gemm(a, b, out_dtype=torch.float32, **kw))
            for p, kw in {1: dict(bn=256, mt=2), 2: dict(split=2), 4: dict(split=4)}.items()}
    assert same == {p: p == parts for p in same}


# the MXFP8 feed-forward node against the layers it stands for: the same bits, dh rounded to bf16 before the activation's gradient, its
# sum whole and in parts; gradients asked for together, with the weights' in main_grad, deferred, and of the input alone
@pytest.mark.parametrize("T,D,F", [(70, 128, 256), (200, 2048, 5632), (300, 768, 2048), (1030, 256, 640)])
@pytest.mark.parametrize("form", ["leaf", "main_grad", "deferred", "input"])
def test_mxfp8_feed_forward_has_the_bits_of_its_layers(T, D, F, form):
    from nanopysche_b200.ops.activation import glu
    from nanopysche_b200.ops.gemm import defer_wgrad, feed_forward_glu, linear, run_deferred_wgrads

    torch.manual_seed(T)
    x0, dy = torch.randn(1, T, D, device="cuda").bfloat16(), torch.randn(1, T, D, device="cuda").bfloat16()
    ws = [(torch.randn(s, device="cuda") * s[1] ** -0.5).bfloat16() for s in ((2 * F, D), (D, F))]

    def grads(layer):
        x, w13, w2 = (t.clone().requires_grad_(form != "input" or t is x0) for t in (x0, *ws))
        for w in (w13, w2):
            w._fp8_recipe = "mxfp8"
            if form in ("main_grad", "deferred"):
                w.main_grad, w._main_grad_dirty = torch.zeros(w.shape, device="cuda"), False
        y, queue = layer(x, w13, w2), []
        if form == "deferred":
            with defer_wgrad(queue):
                y.backward(dy)
            run_deferred_wgrads(queue)
        else:
            y.backward(dy)
        return [y, x.grad] + [getattr(w, "main_grad", w.grad) for w in (w13, w2) if form != "input"]

    got = grads(lambda x, w13, w2: feed_forward_glu(x, w13, w2, "silu"))
    want = grads(lambda x, w13, w2: linear(glu(linear(x, w13), "silu"), w2))
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and len(got) == len(want)
