"""Kernels for a few rows at a time (csrc/skinny.cu) and the head-dim 64 flash kernels, against fp64 PyTorch (GPU only).

bf16 results of sums accumulated in fp32: the distance from the fp64 value is the rounding of the result (2^-9 relative
per value, 0.0017 in the 2-norm of random values) plus, where probabilities are rounded to bf16 before the second product,
as much again per rounding; 6e-3 covers three of them and is far below any indexing mistake."""
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


# rows at the edges of the 8-row tiles and of the dispatch (64 / 65), columns off the 16-row weight tiles, K off the
# 64-wide units and shorter than one round of the warps
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 33, 64, 65])
@pytest.mark.parametrize("N,K", [(2048, 2048), (520, 200), (24, 8), (1000, 72)])
def test_linear_of_a_few_rows(M, N, K):
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(M * N + K)
    x = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K]          # a view with a longer row stride
    w = torch.randn(N, K, device="cuda").bfloat16()
    ref = x.double() @ w.double().t()
    assert rel(gemm(x, w), ref) < 3e-3
    bias, res = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda")
    y = gemm(x, w, alpha=0.5, bias=bias, residual=res, out_dtype=torch.float32)
    assert rel(y, 0.5 * ref + bias.double() + res.double()) < 1e-5
    acc = res.clone()
    gemm(x, w, out=acc, accumulate=True)
    assert rel(acc, ref + res.double()) < 1e-5


def _sdpa64(q, k, v, causal):
    S, T = q.shape[1], k.shape[1]
    m = torch.ones(S, T, dtype=torch.bool, device=q.device).tril(T - S) if causal else None
    return torch.nn.functional.scaled_dot_product_attention(
        q.double().transpose(1, 2), k.double().transpose(1, 2), v.double().transpose(1, 2), attn_mask=m,
        enable_gqa=True).transpose(1, 2)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,S,P,Hq,Hkv,causal", [
    (2, 1, 1, 4, 4, True), (1, 1, 127, 8, 1, True), (3, 1, 2047, 16, 8, True), (1, 1, 4096, 12, 12, True),
    (2, 2, 130, 16, 8, True), (2, 3, 65, 4, 2, False), (2, 8, 33, 4, 4, True), (40, 1, 100, 16, 8, True)])
def test_attention_with_appended_cache(B, S, P, Hq, Hkv, causal, hd):
    from nanopysche_b200.ops.attention import attention_append

    torch.manual_seed(P)
    q = torch.randn(B, S, Hq, hd, device="cuda").bfloat16()
    kv = torch.randn(B, P, 2, Hkv, hd, device="cuda").bfloat16()
    k, v = kv[:, :, 0], kv[:, :, 1]                                        # strided views of one cache
    kn, vn = (torch.randn(B, S, Hkv, hd, device="cuda").bfloat16() for _ in range(2))
    with torch.no_grad():
        o, ko, vo = attention_append(q, k, v, kn, vn, causal=causal)
    assert torch.equal(ko, torch.cat([k, kn], 1)) and torch.equal(vo, torch.cat([v, vn], 1))
    assert rel(o, _sdpa64(q, ko, vo, causal)) < 6e-3


def test_append_under_grad_takes_the_differentiable_path():
    from nanopysche_b200.ops.attention import attention_append

    torch.manual_seed(4)
    leaves = [torch.randn(2, n, h, 64, device="cuda").bfloat16().requires_grad_(True)
              for n, h in ((1, 4), (40, 2), (40, 2), (1, 2), (1, 2))]
    o, ko, vo = attention_append(*leaves)
    g = torch.randn_like(o)
    o.backward(g)
    l64 = [t.detach().double().requires_grad_(True) for t in leaves]
    q, k, v, kn, vn = l64
    ref = _sdpa64(q, torch.cat([k, kn], 1), torch.cat([v, vn], 1), True)
    ref.backward(g.double())
    assert rel(o, ref) < 6e-3 and torch.equal(ko, torch.cat(leaves[1::2], 1)) and torch.equal(vo, torch.cat(leaves[2::2], 1))
    for a, b in zip(leaves, l64):
        assert rel(a.grad, b.grad) < 6e-3


def test_append_of_nothing_and_of_more_batches_than_the_grid_takes():
    from nanopysche_b200.ops.attention import attention_append

    torch.manual_seed(5)
    for B, S in ((2, 0), (65536, 1)):
        q, kn, vn = (torch.randn(B, S, 1, 64, device="cuda").bfloat16() for _ in range(3))
        k, v = (torch.randn(B, 3, 1, 64, device="cuda").bfloat16() for _ in range(2))
        with torch.no_grad():
            o, ko, vo = attention_append(q, k, v, kn, vn)
        assert torch.equal(ko, torch.cat([k, kn], 1)) and torch.equal(vo, torch.cat([v, vn], 1)) and o.shape == q.shape
        if S:
            assert rel(o[-64:], _sdpa64(q[-64:], ko[-64:], vo[-64:], True)) < 6e-3


def test_append_does_not_drop_tangents():
    """Forward-mode derivatives of the flash kernels do not exist: a cached step that carries one says so."""
    from torch.autograd import forward_ad as fwAD

    from nanopysche_b200.ops.attention import attention_append

    ts = [torch.randn(1, n, 4, 64, device="cuda").bfloat16() for n in (1, 40, 40, 1, 1)]
    for i in range(5):
        with fwAD.dual_level(), pytest.raises(NotImplementedError):
            attention_append(*(fwAD.make_dual(t, torch.ones_like(t)) if j == i else t for j, t in enumerate(ts)))
    with fwAD.dual_level(), torch.no_grad():
        assert attention_append(*ts)[1].shape[1] == 41


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,causal", [(1, 128, 128, 2, 2, True), (2, 129, 129, 4, 2, True),
                                                   (1, 100, 300, 4, 2, True), (1, 1, 257, 8, 8, True),
                                                   (3, 777, 777, 6, 3, False), (2, 1000, 1000, 4, 4, True)])
def test_flash_head_dim_64(B, Sq, Sk, Hq, Hkv, causal):
    from nanopysche_b200.ops.attention import attention

    torch.manual_seed(Sq)
    qkv = torch.randn(B, max(Sq, Sk), Hq + 2 * Hkv, 64, device="cuda").bfloat16()
    q = qkv[:, :Sq, :Hq].detach().requires_grad_(True)                      # strided views, as the fused projection gives
    k = qkv[:, :Sk, Hq:Hq + Hkv].detach().requires_grad_(True)
    v = qkv[:, :Sk, Hq + Hkv:].detach().requires_grad_(True)
    o = attention(q, k, v, causal=causal)
    g = torch.randn_like(o)
    o.backward(g)
    q64, k64, v64 = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    r = _sdpa64(q64, k64, v64, causal)
    r.backward(g.double())
    for a, b in ((o, r), (q.grad, q64.grad), (k.grad, k64.grad), (v.grad, v64.grad)):
        assert rel(a, b) < 6e-3


def test_flash_head_dim_64_views_that_need_a_copy():
    """Rows that are not 16-byte aligned, a transposed head dimension, a broadcast head: the same values as from copies."""
    from nanopysche_b200.ops.attention import attention

    torch.manual_seed(3)
    base = torch.randn(2, 70, 4, 68, device="cuda").bfloat16()
    odd = base[..., 2:66]
    tr = torch.randn(2, 70, 64, 4, device="cuda").bfloat16().transpose(2, 3)
    wide = torch.randn(2, 70, 1, 64, device="cuda").bfloat16().expand(2, 70, 4, 64)
    for q, k, v in ((odd, odd, odd), (tr, odd, wide), (odd, wide, wide)):
        o = attention(q, k, v)
        assert torch.equal(o, attention(q.contiguous(), k.contiguous(), v.contiguous()))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,Hkv", [(1, 2), (2, 1), (1, 1)])
def test_flash_keys_of_a_longer_buffer(B, Hkv, hd):
    """k is the start of a longer buffer, v a tensor of its own: with a batch or head count of 1 both count as contiguous
    although their strides differ. Forward and backward give what copies give."""
    from nanopysche_b200.ops.attention import attention

    torch.manual_seed(hd)
    q = torch.randn(B, 40, 4, hd, device="cuda").bfloat16()
    buf = torch.randn(B, 300, Hkv, hd, device="cuda").bfloat16()
    v = torch.randn(B, 200, Hkv, hd, device="cuda").bfloat16()
    wide = torch.randn(B, 200, 3 * Hkv, hd, device="cuda").bfloat16()
    g = torch.randn_like(q)

    def grads(k, v):
        leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
        o = attention(*leaves)
        return [o, *torch.autograd.grad(o, leaves, g)]

    for kk, vv in ((buf[:, :200], v), (v, buf[:, :200]), (wide[:, :, :Hkv], v), (buf[:, 50:250], wide[:, :, Hkv:2 * Hkv])):
        for a, b in zip(grads(kk, vv), grads(kk.clone(memory_format=torch.contiguous_format),
                                             vv.clone(memory_format=torch.contiguous_format))):
            assert torch.equal(a, b)


# the few-row kernel reads all of x again for every 16 columns: with many columns the tile kernels take over as rows are added
@pytest.mark.parametrize("M,N,K,few", [(1, 32000, 1024, True), (8, 32000, 1024, True), (16, 32000, 1024, False),
                                       (64, 32000, 1024, False), (64, 2048, 2048, True), (65, 2048, 2048, False)])
def test_few_row_kernel_where_it_is_the_faster_one(M, N, K, few):
    from nanopysche_b200.ops.gemm import gemm

    torch.manual_seed(M)
    x, w = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    out = gemm(x, w)
    assert rel(out, x.double() @ w.double().t()) < 3e-3
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        gemm(x, w, out=out)
        torch.cuda.synchronize()
    assert any("skinny" in e.key for e in p.key_averages()) == few
