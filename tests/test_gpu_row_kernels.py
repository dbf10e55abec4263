"""Row-wise and token-wise kernels at the edges of their blocking, against fp64 PyTorch (GPU only). Tolerances: one rounding
of the result to bf16 (2-norm 0.0017) plus fp32 sums, doubled; fp32 results 1e-5."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b.double()).norm() / (b.double().norm() + 1e-30)).item()


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
