"""Attention backward where its buffers turn over: one, two and more blocks per tile, ragged ends, groups of query heads, both
head dimensions, two and four threads per score row, against fp64 PyTorch (GPU only). Tolerance: P, dS and the results are
rounded to bf16 (2-norm 0.0017 each, two of them in a chain with the rounded inputs' products), doubled."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,split", [(128, 2), (128, 4), (64, 2)])
@pytest.mark.parametrize("B,S,hq,hkv,causal", [(1, 128, 2, 1, True), (2, 130, 3, 1, False), (1, 384, 2, 2, False),
                                               (1, 640, 6, 2, True), (1, 1000, 2, 1, True)])
def test_backward(B, S, hq, hkv, causal, hd, split):
    from nanopysche_b200.ops.attention import flash_bwd, flash_fwd

    torch.manual_seed(S + hd)
    q, do = (torch.randn(B, S, hq, hd, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, S, hkv, hd, device="cuda").bfloat16() for _ in range(2))
    o, lse = flash_fwd(q, k, v, causal=causal)
    got = flash_bwd(q, k, v, o, do, lse, causal=causal, split=split)
    q64, k64, v64 = (t.double().requires_grad_(True) for t in (q, k, v))
    kk, vv = (t.repeat_interleave(hq // hkv, 2).transpose(1, 2) for t in (k64, v64))
    s = q64.transpose(1, 2) @ kk.transpose(2, 3) * hd ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(S, S, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    (s.softmax(-1) @ vv).transpose(1, 2).backward(do.double())
    for a, b in zip(got, (q64.grad, k64.grad, v64.grad)):
        assert ((a.double() - b).norm() / b.norm()).item() < 8e-3
