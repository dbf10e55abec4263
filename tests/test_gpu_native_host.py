"""The native host module (csrc/host.cpp): what its autograd nodes save, refuse and leave to others, and the attention node against
the ops it stands for (GPU only). bf16 results against the separate nodes: the same kernels, so the same bits."""
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


def _randn(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


# heads of 64 and 128, sequence off the blocks, a position offset, positions of their own, per-head norms, gradients that are
# broadcast or cut from a wider tensor
@pytest.mark.parametrize("B,S,hq,hkv,hd,causal,norm", [(1, 1, 2, 1, 64, True, False), (2, 130, 4, 4, 64, True, False),
                                                       (3, 77, 4, 2, 128, False, False), (2, 257, 4, 2, 128, True, True),
                                                       (1, 300, 16, 8, 128, False, True)])
@pytest.mark.parametrize("grad", ["dense", "expanded", "cut"])
def test_attention_node_is_rotation_and_attention(B, S, hq, hkv, hd, causal, norm, grad):
    from nanopysche_b200.ops import attention as A
    from nanopysche_b200.ops import rope as R

    torch.manual_seed(S)
    qkv = _randn(B, S, (hq + 2 * hkv) * hd).requires_grad_(True)
    cos, sin = R.rope_tables(S + 9, hd, device="cuda")
    ids = torch.randint(0, S + 9, (B, S), device="cuda") if S % 2 else None
    pos = 0 if ids is not None else 5
    norms = [torch.nn.LayerNorm(hd, device="cuda") for _ in range(2)] if norm else [None, None]
    for m in norms:
        if m is not None:
            torch.nn.init.normal_(m.weight, 1.0, 0.2), torch.nn.init.normal_(m.bias, 0.0, 0.2)
    par = [p for m in norms if m is not None for p in m.parameters()]
    dy = {"dense": _randn(B, S, hq * hd), "expanded": _randn(hq * hd).expand(B, S, -1), "cut": _randn(B, S, hq * hd + 8)[..., 8:]}[grad]
    o = A.qkv_attention(qkv, cos, sin, hq, hkv, hd, pos, ids, causal, *norms)
    got = torch.autograd.grad(o, [qkv, *par], dy)
    split = R.qkv_rope(qkv, cos, sin, hq, hkv, hd, pos, ids) if not norm else R.qkv_norm_rope(qkv, *norms, cos, sin, hq, hkv, pos, ids)
    want_o = A.attention(*split, causal=causal).reshape(B, S, hq * hd)
    want = torch.autograd.grad(want_o, [qkv, *par], dy)
    assert torch.equal(o, want_o) and torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):          # atomic sums over the heads of a kind
        assert rel(a, b) < 1e-5


def test_attention_node_leaves_other_forms():
    from nanopysche_b200.ops import attention as A
    from nanopysche_b200.ops import rope as R

    cos, sin = R.rope_tables(32, 32, device="cuda")
    assert A.qkv_attention(_randn(1, 32, 6 * 32), cos, sin, 2, 2, 32) is None               # head dimension
    cos, sin = R.rope_tables(32, 128, device="cuda")
    assert A.qkv_attention(_randn(1, 32, 4 * 128).float(), cos, sin, 2, 1, 128) is None     # dtype
    wide = _randn(2, 40, 4 * 128)[:, :32]                                                   # rows of a longer buffer
    assert A.qkv_attention(wide, cos, sin, 2, 1, 128) is None


def test_nodes_save_through_hooks_and_refuse_transforms():
    from nanopysche_b200.ops.gemm import linear
    from nanopysche_b200.ops.norm import rms_norm

    x, w, g = _randn(2, 70, 128).requires_grad_(True), _randn(64, 128).requires_grad_(True), torch.rand(128, device="cuda", requires_grad=True)
    want = torch.autograd.grad(linear(rms_norm(x, g), w), [x, w, g], torch.ones(2, 70, 64, device="cuda").bfloat16())
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.cuda()):
        y = linear(rms_norm(x, g), w)
    assert torch.Size([64, 128]) in packed and torch.Size([2, 70, 128]) in packed
    got = torch.autograd.grad(y, [x, w, g], torch.ones(2, 70, 64, device="cuda").bfloat16())
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x))
        with pytest.raises(RuntimeError):
            linear(dual, w)
        with pytest.raises(RuntimeError):
            rms_norm(dual, g)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: linear(t, w.detach()))(x.detach())
    with torch.autograd.graph.save_on_cpu():
        y = linear(x, w)
    with torch.no_grad():
        w.add_(1.0)
    assert linear(x, w).grad_fn is not None
    y = linear(x, w)
    with torch.no_grad():
        w.mul_(2.0)
    with pytest.raises(RuntimeError, match="inplace"):      # a saved weight that was written since
        y.sum().backward()


def test_errors_are_the_ops_own():
    from nanopysche_b200.ops import _lib
    from nanopysche_b200.ops.gemm import gemm, linear

    with pytest.raises(AssertionError, match="contraction mismatch 128 vs 120"):
        linear(_randn(4, 128), _randn(64, 120))
    with pytest.raises(AssertionError, match="bf16"):
        gemm(_randn(4, 128), torch.randn(64, 128, device="cuda"))
    with pytest.raises(_lib.KernelError, match="code 1"):
        gemm(_randn(200, 136)[:, :129], _randn(64, 136)[:, 1:130])      # rows of B off the 16-byte boundaries
    n = _lib.LAUNCHES
    linear(_randn(300, 128), _randn(64, 128))
    assert _lib.LAUNCHES == n + 1


@pytest.mark.parametrize("need_x", [True, False])
def test_main_grad_and_deferred_weight_gradients(need_x):
    from nanopysche_b200.ops.gemm import defer_wgrad, linear, run_deferred_wgrads

    torch.manual_seed(0)
    x, dy = _randn(300, 256).requires_grad_(need_x), _randn(300, 512)
    w = _randn(512, 256).requires_grad_(True)
    want = (dy.float().t() @ x.detach().float())
    w.main_grad, done = torch.full((512, 256), 7.0, device="cuda"), []
    w._main_grad_dirty, w._grad_ready_cb = False, done.append
    linear(x, w).backward(dy)
    assert rel(w.main_grad, want) < 2e-5 and w._main_grad_dirty and done == [w] and w.grad is None      # written over
    linear(x, w).backward(dy)
    assert rel(w.main_grad, 2 * want) < 2e-5                                                            # added
    w._main_grad_dirty, queue = False, []
    with defer_wgrad(queue):
        linear(x, w).backward(dy)
    assert len(queue) == 1 and rel(w.main_grad, 2 * want) < 2e-5 and (x.grad is not None) == need_x
    run_deferred_wgrads(queue)
    assert rel(w.main_grad, want) < 2e-5
