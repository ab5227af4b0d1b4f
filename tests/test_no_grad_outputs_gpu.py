"""Forward passes without gradients leave out what only the backward reads; their results are those of the training forward."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_swiglu_gemm_without_gradients():
    from archscale_b200.ops import gemm
    torch.manual_seed(10)
    x = torch.randn(520, 256, device="cuda").bfloat16()
    w = torch.nn.Parameter((torch.randn(2 * 136, 256, device="cuda") / 16).bfloat16())
    y = gemm.linear_swiglu(x, w)
    assert y is not None and y.requires_grad
    with torch.no_grad():
        y0 = gemm.linear_swiglu(x, w)
    assert torch.equal(y, y0)
    g, u = (x.double() @ w.detach().double().t()).chunk(2, -1)
    r = torch.nn.functional.silu(g) * u
    assert float((y0.double() - r).norm()) <= 1e-2 * float(r.norm())


@pytest.mark.parametrize("rows", [512, 777])
def test_linear_cross_entropy_without_gradients(rows):
    from archscale_b200.ops.cross_entropy import fused_linear_cross_entropy
    torch.manual_seed(11)
    h = torch.randn(rows, 256, device="cuda").bfloat16()
    w = torch.nn.Parameter((torch.randn(1000, 256, device="cuda") * 0.05).bfloat16())
    t = torch.randint(0, 1000, (rows,), device="cuda")
    t[::7] = -100
    loss = fused_linear_cross_entropy(h, w, t)
    with torch.no_grad():
        loss0 = fused_linear_cross_entropy(h, w, t)
    assert torch.equal(loss, loss0) and not loss0.requires_grad
    loss.backward()
    ref = torch.autograd.grad(torch.nn.functional.cross_entropy(h.double() @ (wd := w.detach().double().requires_grad_()).t(), t), wd)[0]
    assert float((w.grad.double() - ref).norm()) <= 1e-2 * float(ref.norm())
