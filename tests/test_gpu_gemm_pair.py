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
