"""One-group SSD scan: the skip factors D in every shape that holds one number per head."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(4,), (4, 1), (1, 4), (2, 2), (1, 1, 4, 1)])
def test_skip_factor_shapes(shape, dtype):
    from archscale_b200.ops.ssd import ssd_scan
    mk = lambda *s: torch.randn(*s, device="cuda").to(dtype)
    x, dt, A = mk(1, 70, 4, 64), torch.rand(1, 70, 4, device="cuda") * 0.3, -torch.rand(4, device="cuda") - 0.1
    B, C, D = mk(1, 70, 1, 16), mk(1, 70, 1, 16), torch.randn(4, device="cuda")
    flat, other = D.clone().requires_grad_(True), D.clone().reshape(shape).requires_grad_(True)
    y0, y1 = ssd_scan(x, dt, A, B, C, flat), ssd_scan(x, dt, A, B, C, other)
    assert torch.equal(y0, y1)
    g = torch.randn_like(y0)
    d0, d1 = torch.autograd.grad(y0, flat, g)[0], torch.autograd.grad(y1, other, g)[0]
    assert d1.shape == other.shape and torch.equal(d0, d1.reshape(4))
